// Phase 1 of a column: level bins and per-band opacity terms into shared memory.
// Restates the set-up loops of code/optcv.f90:103-124,182-247 and
// code/optci.f90:113-131,182-220 plus the Planck boundary terms of
// code/sfluxi.f90:51-62 and code/gfluxi.f90:69-87.
#pragma once
#include "rt_column.cuh"
#include "rt_fastmath.cuh"

namespace mgcm {

// Input checks folded into the staging, which reads nearly every input value
// anyway.  A kernel of its own, a thread per column walking 35 KB of strided
// values, was bound by its serial reads; without it a validated call takes
// 0.79 -> 0.27 ms for 60 x 24 columns, 4.51 -> 3.00 ms for 8,640 x 36
// (MIXED), 14.4 -> 13.4 ms for 64,800 x 24 (FP64).  A value costs one multiply-add: v * 0 is 0 for a finite v and NaN
// otherwise, and NaN stays in the sum.  With V false nothing is checked.
template <bool V>
struct Check {
    double acc = 0.0;
    bool neg = false, temp = false;
    __device__ __forceinline__ void finite(double v) {
        if (V) acc = fma(v, 0.0, acc);
    }
    __device__ __forceinline__ void pressure(double v) {   // NaN, Inf or <= 0
        if (V) {
            finite(v);
            neg |= !(v > 0.0);
        }
    }
    __device__ __forceinline__ void temperature(double t) {   // outside the Planck table
        if (V) {
            finite(t);
            const double x = __dsub_rn(__dmul_rn(t, 10.0), 499.0);
            temp |= !(x >= 1.0 && x < 8502.0);
        }
    }
    __device__ __forceinline__ void report(uint32_t *status) {
        if (V) {
            const uint32_t bad = (acc != 0.0 || neg ? ST_NONFINITE : 0u) | (temp ? ST_TEMP : 0u);
            if (bad) atomicOr(status, bad);
        }
    }
};

// A layer the solves' fast arithmetic may take: |COSBAR| < 1, a numerator of
// the single-scattering albedo that is 0 or in [2^-300, 2^300).  Any physical
// layer is; a column with another one goes through the general solve.
__device__ __forceinline__ bool usual_layer(double cosb, double wnum) {
    return fabs(cosb) < 1.0 && (wnum == 0.0 || (wnum > 0.0 && !out_of_range(wnum)));
}

// Level item k (2..LEV+1) of column c: bins, U, DPR and the TAUREF ratios.
// With V the item checks the level's inputs; item 2 also level 1 and the
// column's scalars, and the items share the column's 119 DETAU.
template <bool V>
__device__ inline void stage_level(const SegDev &sg, int c, const RtConst &K, ColSmem &s, int k,
                                   uint32_t *status) {
    const int L = sg.L, LEV = 2 * L + 3, LEV1 = LEV + 1;
    const double *plev = sg.plev + (size_t)c * LEV;
    const double *tlev = sg.tlev + (size_t)c * LEV;
    const double *pmid = sg.pmid + (size_t)c * LEV;
    const double *tmid = sg.tmid + (size_t)c * LEV;
    const double *qh2o = sg.qh2o + (size_t)c * LEV;
    const double *tauref = sg.tauref + (size_t)c * LEV1;
    const double *db = sg.dust_band;   // prescribed dust: band constants
    const double *qxref = db ? nullptr : sg.qextrefdst + (size_t)c * LEV1;
    const double *qxv = db ? nullptr : sg.qxvdst + (size_t)c * D_NV * LEV1;
    const bool cld = sg.taurefcld != nullptr;
    const double *taucld = cld ? sg.taurefcld + (size_t)c * LEV1 : nullptr;
    const double *qxcld = cld ? sg.qextrefcld + (size_t)c * LEV1 : nullptr;

    {
        if (k <= LEV) {
            int mt, mp, nh;
            double wr, lk[4];
            tpindex_dev(K, pmid[k - 1], tmid[k - 1], qh2o[k - 1], mt, mp, nh, wr, lk);
            const int nh1 = nh < D_NH ? nh + 1 : D_NH;   // WRATIO = 0 when NH2O = 10
            KLevel &kl = s.klev[k];
            kl.kofs = (((mt - 1) * D_NP + (mp - 1)) * D_NH + (nh - 1)) * D_NGK;
            kl.kdh = (nh1 - nh) * D_NGK;
            kl.wr = wr;
            kl.lk[0] = lk[0];
            kl.lk[1] = lk[1];
            kl.lk[2] = lk[2];
            kl.lk[3] = lk[3];
            kl.same = 0;
            if ((k & 1) == 0 && k >= 4 && pmid[k - 1] == pmid[k - 2] && tmid[k - 1] == tmid[k - 2]) {
                if (qh2o[k - 1] == qh2o[k - 2])
                    kl.same = SAME_VALUE;
                else if (water_bin(K, qh2o[k - 2]) == nh)
                    kl.same = SAME_CORNERS;
            }
            const double dpr = plev[k - 1] - plev[k - 2];
            s.dpr[k] = dpr;
            kl.u = 3.51e22 * dpr;
            s.tref_v[k] = tauref[k - 1] / (db ? db[NREFV_IDX] : qxv[(size_t)(NREFV_IDX)*LEV1 + k - 1]);
            s.tref_i[k] = tauref[k - 1] / (db ? db[NREFV_IDX] : qxref[k - 1]);
            s.tref_c[k] = cld ? taucld[k - 1] / qxcld[k - 1] : 0.0 / 1.0;
            if (k == 2) *s.odd = 0;   // the band items come after a barrier
        } else {
            s.tref_i[k] = db ? 0.0 : tauref[k - 1];
            s.tref_c[k] = cld ? taucld[k - 1] : 0.0;
        }
    }
    if (V) {
        Check<V> chk;
        auto level = [&](int i) {   // values of level i + 1
            if (i < LEV) {
                chk.pressure(plev[i]);
                chk.pressure(pmid[i]);
                chk.temperature(tlev[i]);
                chk.finite(tmid[i]);
                chk.finite(qh2o[i]);
            }
            if (i < LEV || !db) chk.finite(tauref[i]);   // TAUREF(LEV+1) is 0 with prescribed dust
            if (!db) chk.finite(qxref[i]);
            if (cld) {
                chk.finite(taucld[i]);
                chk.finite(qxcld[i]);
            }
        };
        level(k - 1);
        if (k == 2) {
            level(0);
            chk.finite(sg.acosz[c]);
            chk.finite(sg.als[c]);
            chk.finite(sg.albi[c]);
            chk.finite(sg.pcol[c]);
        }
        for (int i = k - 2; i < D_NV * D_NG; i += LEV1 - 1) chk.finite(sg.detau[(size_t)c * (D_NV * D_NG) + i]);
        chk.report(status);
    }
}

// Band items of a column: nitem_v = (NL+1)*7 visible (layer l = 0..NL: level 2
// for l = 0), nitem_i = (NL+1)*5 IR with the Planck terms, then 5 IR boundary
// items.  Needs every level item of the column staged first.
__device__ __forceinline__ int stage_band_items(int L) { return (L + 2) * (D_NV + D_NI) + D_NI; }

// With V the items check every value of the band arrays: layer item l its
// levels, item 0 also level 1 and item NL level LEV+1.
template <bool V>
__device__ inline void stage_band(const SegDev &sg, int c, const RtConst &K,
                                  const double *__restrict__ planck, ColSmem &s, int it,
                                  uint32_t *status) {
    const int L = sg.L, NL = L + 1, LEV = 2 * L + 3, LEV1 = LEV + 1;
    const double *tlev = sg.tlev + (size_t)c * LEV;
    const bool cld = sg.taurefcld != nullptr;
    const int nitem_v = (NL + 1) * D_NV, nitem_i = (NL + 1) * D_NI;
    Check<V> chk;
    {
        if (it < nitem_v) {
            const int l = it / D_NV, nw = it % D_NV + 1;
            // dust properties of level k at qx[(k - 1) * ks] (ks = 0: band constants)
            const double *db = sg.dust_band;
            const int ks = db ? 0 : 1;
            const double *qx = db ? db + nw - 1 : sg.qxvdst + ((size_t)c * D_NV + nw - 1) * LEV1;
            const double *qs = db ? db + D_NV + nw - 1 : sg.qsvdst + ((size_t)c * D_NV + nw - 1) * LEV1;
            const double *gv = db ? db + 2 * D_NV + nw - 1 : sg.gvdst + ((size_t)c * D_NV + nw - 1) * LEV1;
            const double *qxc = cld ? sg.qxvcld + ((size_t)c * D_NV + nw - 1) * LEV1 : nullptr;
            const double *qsc = cld ? sg.qsvcld + ((size_t)c * D_NV + nw - 1) * LEV1 : nullptr;
            const double *gc = cld ? sg.gvcld + ((size_t)c * D_NV + nw - 1) * LEV1 : nullptr;
            const double tr0 = K.tauray[nw - 1];
            auto check = [&](int i) {
                if (V) {
                    if (!db) {
                        chk.finite(qx[i]);
                        chk.finite(qs[i]);
                        chk.finite(gv[i]);
                    }
                    if (cld) {
                        chk.finite(qxc[i]);
                        chk.finite(qsc[i]);
                        chk.finite(gc[i]);
                    }
                }
            };
            auto lvl = [&](int k, double &tr, double &tl, double &tc, double &g1, double &g2) {
                tr = tr0 * s.dpr[k];
                const double taeros = s.tref_v[k] * qx[(k - 1) * ks];
                const double tcloud = s.tref_c[k] * (cld ? qxc[k - 1] : 0.0);
                s.ray(k, nw) = tr + taeros + tcloud;
                tl = s.tref_v[k] * qs[(k - 1) * ks];
                tc = s.tref_c[k] * (cld ? qsc[k - 1] : 0.0);
                g1 = gv[(k - 1) * ks];
                g2 = cld ? gc[k - 1] : 0.0;
                check(k - 1);
            };
            bool usual = true;
            double tra, tla, tca, ga, gca;
            if (l == 0) {
                lvl(2, tra, tla, tca, ga, gca);
                check(0);
            } else if (l <= L) {
                const int k = 2 * l + 1;
                double trb, tlb, tcb, gb, gcb;
                lvl(k, tra, tla, tca, ga, gca);
                lvl(k + 1, trb, tlb, tcb, gb, gcb);
                const double cb = (ga * tla + gb * tlb + gca * tca + gcb * tcb) / (tra + trb + tla + tlb + tca + tcb);
                s.lay_v[l * D_NV + nw - 1].cosb = cb;
                s.lay_v[l * D_NV + nw - 1].cbs = cb / (1.0 + cb);   // code/getdetau.f90:29-56
                const double wn = tla + tlb + tca + tcb + (tra + trb) * R4(0.9999);
                s.lay_v[l * D_NV + nw - 1].wnum = wn;
                usual = usual_layer(cb, wn);
            } else {
                const int k = LEV;
                lvl(k, tra, tla, tca, ga, gca);
                const double cb = (ga * tla + gca * tca) / (tra + tla + tca);
                s.lay_v[l * D_NV + nw - 1].cosb = cb;
                s.lay_v[l * D_NV + nw - 1].cbs = cb / (1.0 + cb);
                const double wn = tla + tca + tra * R4(0.9999);
                s.lay_v[l * D_NV + nw - 1].wnum = wn;
                usual = usual_layer(cb, wn);
                check(LEV);
            }
            if (!usual) atomicOr(s.odd, 1 << (nw - 1));
        } else if (it < nitem_v + nitem_i) {
            const int j = it - nitem_v;
            const int l = j / D_NI, nw = j % D_NI + 1;
            const double *db = sg.dust_band;
            const int ks = db ? 0 : 1;
            const double *qx = db ? db + 3 * D_NV + nw - 1 : sg.qxidst + ((size_t)c * D_NI + nw - 1) * LEV1;
            const double *qs = db ? db + 3 * D_NV + D_NI + nw - 1
                                  : sg.qsidst + ((size_t)c * D_NI + nw - 1) * LEV1;
            const double *gi = db ? db + 3 * D_NV + 2 * D_NI + nw - 1
                                  : sg.gidst + ((size_t)c * D_NI + nw - 1) * LEV1;
            const double *qxc = cld ? sg.qxicld + ((size_t)c * D_NI + nw - 1) * LEV1 : nullptr;
            const double *qsc = cld ? sg.qsicld + ((size_t)c * D_NI + nw - 1) * LEV1 : nullptr;
            const double *gc = cld ? sg.gicld + ((size_t)c * D_NI + nw - 1) * LEV1 : nullptr;
            auto ext = [&](int k) {   // TAEROS, TCLOUD at level k <= LEV
                s.ext(k, nw).x = s.tref_i[k] * qx[(k - 1) * ks];
                s.ext(k, nw).y = s.tref_c[k] * (cld ? qxc[k - 1] : 0.0);
            };
            auto check = [&](int i) {
                if (V) {
                    if (!db) {
                        chk.finite(qx[i]);
                        chk.finite(qs[i]);
                        chk.finite(gi[i]);
                    }
                    if (cld) {
                        chk.finite(qxc[i]);
                        chk.finite(qsc[i]);
                        chk.finite(gc[i]);
                    }
                }
            };
            if (l == 0) {
                ext(2);
                check(0);
                check(1);
            } else {
                const int k = 2 * l + 1;
                ext(k);
                if (k + 1 <= LEV) ext(k + 1);
                check(k - 1);
                check(k);
                const double tla = s.tref_i[k] * qs[(k - 1) * ks], tlb = s.tref_i[k + 1] * qs[k * ks];
                const double tca = s.tref_c[k] * (cld ? qsc[k - 1] : 0.0);
                const double tcb = s.tref_c[k + 1] * (cld ? qsc[k] : 0.0);
                const double tauac = tla + tlb + tca + tcb;
                s.lay_i[l * D_NI + nw - 1].wnum = tauac;
                double cb = 0.0;
                if (tauac > 0.0)
                    cb = (gi[(k - 1) * ks] * tla + gi[k * ks] * tlb + (cld ? gc[k - 1] : 0.0) * tca +
                          (cld ? gc[k] : 0.0) * tcb) /
                         (tla + tlb + tca + tcb);
                s.lay_i[l * D_NI + nw - 1].cosb = cb;
                // Planck source terms (gfluxi.f90:219-239)
                const int na = planck_index(l < NL ? tlev[2 * l - 1] : tlev[2 * l + 1 - 1], status);
                const int nb = planck_index(l < NL ? tlev[2 * l + 2 - 1] : tlev[2 * l - 1], status);
                const double pa = planck[(na - 1) * D_NI + nw - 1], pb = planck[(nb - 1) * D_NI + nw - 1];
                const double pd = l < NL ? pb - pa : pa - pb;
                s.lay_i[l * D_NI + nw - 1].pdif = pd;
                s.lay_i[l * D_NI + nw - 1].b0 = l < NL ? pa : pb;
                if (!usual_layer(cb, tauac) || (pd != 0.0 && out_of_range(pd)))
                    atomicOr(s.odd, 1 << (D_NV + nw - 1));
            }
        } else {
            // IR boundary terms (sfluxi.f90:51-62)
            const int nw = it - nitem_v - nitem_i + 1;
            const int nts = planck_index(tlev[LEV - 1], status);
            const int ntt = planck_index(tlev[2 - 1], status);
            s.bsurf_i[nw - 1] = (1.0 - sg.albi[c]) * planck[(nts - 1) * D_NI + nw - 1];
            s.pltop_i[nw - 1] = planck[(ntt - 1) * D_NI + nw - 1];
        }
    }
    chk.report(status);
}

// The whole column by one CTA (the fused kernel).
__device__ inline void stage_column(const SegDev &sg, int c, const RtConst &K,
                                    const double *__restrict__ planck, ColSmem &s,
                                    uint32_t *status) {
    const int LEV1 = 2 * sg.L + 4;
    for (int k = 2 + (int)threadIdx.x; k <= LEV1; k += blockDim.x) stage_level<false>(sg, c, K, s, k, status);
    __syncthreads();
    const int n = stage_band_items(sg.L);
    for (int it = threadIdx.x; it < n; it += blockDim.x) stage_band<false>(sg, c, K, planck, s, it, status);
}

}  // namespace mgcm

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

// Record of layer l (0..NL; 0: level 2 only) of a band b of a column: 0..6
// visible, 7..11 IR with the Planck terms, layer 0 of the IR bands also the
// boundary terms.  Needs every level item of the column staged first.  Lanes
// along the layers read each input array contiguously and write whole records.
// With V the items check every value of the band arrays: a layer item its
// levels, layer 0 also level 1 and layer NL level LEV+1.
template <bool V>
__device__ inline void stage_band(const SegDev &sg, int c, const RtConst &K,
                                  const double *__restrict__ planck, ColSmem &s, int b, int l,
                                  uint32_t *status) {
    const int L = sg.L, NL = L + 1, LEV = 2 * L + 3, LEV1 = LEV + 1;
    const bool cld = sg.taurefcld != nullptr;
    Check<V> chk;
    const bool vis = b < D_NV;
    const int nb = vis ? D_NV : D_NI, w = vis ? b : b - D_NV;   // 0-based band of the family
    // dust properties of level k at q[(k - 1) * ks] (ks = 0: band constants)
    const double *db = sg.dust_band;
    const int ks = db ? 0 : 1;
    const size_t row = ((size_t)c * nb + w) * LEV1;
    const double *qx, *qs, *qg, *cx = nullptr, *cs = nullptr, *cg = nullptr;
    if (vis) {
        qx = db ? db + w : sg.qxvdst + row;
        qs = db ? db + D_NV + w : sg.qsvdst + row;
        qg = db ? db + 2 * D_NV + w : sg.gvdst + row;
        if (cld) { cx = sg.qxvcld + row; cs = sg.qsvcld + row; cg = sg.gvcld + row; }
    } else {
        qx = db ? db + 3 * D_NV + w : sg.qxidst + row;
        qs = db ? db + 3 * D_NV + D_NI + w : sg.qsidst + row;
        qg = db ? db + 3 * D_NV + 2 * D_NI + w : sg.gidst + row;
        if (cld) { cx = sg.qxicld + row; cs = sg.qsicld + row; cg = sg.gicld + row; }
    }
    struct Lv {
        double qx, qs, g, cx, cs, cg;
    };
    auto read = [&](int k) {   // level k <= LEV1
        Lv v;
        v.qx = qx[(k - 1) * ks];
        v.qs = qs[(k - 1) * ks];
        v.g = qg[(k - 1) * ks];
        v.cx = cld ? cx[k - 1] : 0.0;
        v.cs = cld ? cs[k - 1] : 0.0;
        v.cg = cld ? cg[k - 1] : 0.0;
        chk.finite(v.qx);
        chk.finite(v.qs);
        chk.finite(v.g);
        chk.finite(v.cx);
        chk.finite(v.cs);
        chk.finite(v.cg);
        return v;
    };
    const int ka = l ? 2 * l + 1 : 2;   // the item's first level
    const Lv A = read(ka);
    Lv B = {};
    if (l) B = read(ka + 1);             // the layer's second level; LEV+1 for l = NL
    else if (V) read(1);
    bool usual = true;
    if (vis) {
        const double tr0 = K.tauray[w];
        VisLayer r;
        r.cosb = r.wnum = r.cbs = r.pad = 0.0;
        const double tra = tr0 * s.dpr[ka];
        const double raya = tra + s.tref_v[ka] * A.qx + s.tref_c[ka] * A.cx;
        const double tla = s.tref_v[ka] * A.qs, tca = s.tref_c[ka] * A.cs;
        r.ray[0] = l ? raya : 0.0;
        r.ray[1] = l ? 0.0 : raya;
        if (l && l <= L) {
            const int kb = ka + 1;
            const double trb = tr0 * s.dpr[kb];
            r.ray[1] = trb + s.tref_v[kb] * B.qx + s.tref_c[kb] * B.cx;
            const double tlb = s.tref_v[kb] * B.qs, tcb = s.tref_c[kb] * B.cs;
            r.cosb = (A.g * tla + B.g * tlb + A.cg * tca + B.cg * tcb) / (tra + trb + tla + tlb + tca + tcb);
            r.wnum = tla + tlb + tca + tcb + (tra + trb) * R4(0.9999);
        } else if (l) {
            r.cosb = (A.g * tla + A.cg * tca) / (tra + tla + tca);
            r.wnum = tla + tca + tra * R4(0.9999);
        }
        if (l) {
            r.cbs = r.cosb / (1.0 + r.cosb);   // code/getdetau.f90:29-56
            usual = usual_layer(r.cosb, r.wnum);
        }
        s.vis(l, w + 1) = r;
    } else {
        const double *tlev = sg.tlev + (size_t)c * LEV;
        IrLayer r;
        r.cosb = r.wnum = r.b0 = r.pdif = 0.0;
        const double2 exta = make_double2(s.tref_i[ka] * A.qx, s.tref_c[ka] * A.cx);   // TAEROS, TCLOUD
        r.ext[0] = exta;
        r.ext[1] = l ? make_double2(0.0, 0.0) : exta;
        if (l) {
            const int kb = ka + 1;
            if (kb <= LEV) r.ext[1] = make_double2(s.tref_i[kb] * B.qx, s.tref_c[kb] * B.cx);
            const double tla = s.tref_i[ka] * A.qs, tlb = s.tref_i[kb] * B.qs;
            const double tca = s.tref_c[ka] * A.cs, tcb = s.tref_c[kb] * B.cs;
            const double tauac = tla + tlb + tca + tcb;
            if (tauac > 0.0)
                r.cosb = (A.g * tla + B.g * tlb + A.cg * tca + B.cg * tcb) / (tla + tlb + tca + tcb);
            r.wnum = tauac;
            // Planck source terms (gfluxi.f90:219-239)
            const int na = planck_index(l < NL ? tlev[2 * l - 1] : tlev[2 * l + 1 - 1], status);
            const int nt = planck_index(l < NL ? tlev[2 * l + 2 - 1] : tlev[2 * l - 1], status);
            const double pa = planck[(na - 1) * D_NI + w], pb = planck[(nt - 1) * D_NI + w];
            r.pdif = l < NL ? pb - pa : pa - pb;
            r.b0 = l < NL ? pa : pb;
            usual = usual_layer(r.cosb, tauac) && (r.pdif == 0.0 || !out_of_range(r.pdif));
        } else {
            // IR boundary terms (sfluxi.f90:51-62)
            const int nts = planck_index(tlev[LEV - 1], status);
            const int ntt = planck_index(tlev[2 - 1], status);
            s.bsurf_i[w] = (1.0 - sg.albi[c]) * planck[(nts - 1) * D_NI + w];
            s.pltop_i[w] = planck[(ntt - 1) * D_NI + w];
        }
        s.ir(l, w + 1) = r;
    }
    if (!usual) atomicOr(s.odd, 1 << b);
    chk.report(status);
}

// The whole column by one CTA (the fused kernel).
__device__ inline void stage_column(const SegDev &sg, int c, const RtConst &K,
                                    const double *__restrict__ planck, ColSmem &s,
                                    uint32_t *status) {
    const int LEV1 = 2 * sg.L + 4;
    for (int k = 2 + (int)threadIdx.x; k <= LEV1; k += blockDim.x) stage_level<false>(sg, c, K, s, k, status);
    __syncthreads();
    const int n = (sg.L + 2) * (D_NV + D_NI);
    for (int it = threadIdx.x; it < n; it += blockDim.x)
        stage_band<false>(sg, c, K, planck, s, it / (sg.L + 2), it % (sg.L + 2), status);
}

}  // namespace mgcm

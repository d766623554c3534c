// Aerosol optics on the device: the per-level dust and water-ice optical
// properties that COMP3 prepares for OPTCV/OPTCI, from tracer mixing ratios
// (code/comp3.f:592-630):
//   active dust  OPT_DST  code/opt_dst.f:55-161
//   prescribed   INI_OPTDST band constants (code/ini_optdst.f:29-51,
//                code/setrad.f90:132-155) with TAUREF given (FILLTAUCUM)
//   water ice    OPT_CLD  code/opt_cld.f:55-188
// Per layer: a lognormal size distribution from the mass and number mixing
// ratios, bin weights from DERF differences over the 20 radiative-transfer
// bins, band sums of the REAL*4 Mie tables for the layer's two levels, and
// TAUREF.  Built with --fmad=false; powers, logs, exps and DERF come from
// include/mgcm_rt_math.h, so the results equal the CPU oracle's bit for bit.
//
// One warp per family and 16 layers (32 levels) of a column.  A lane per layer
// applies the routines' thresholds and computes the size parameters; then the
// lanes take (layer, bin edge) items: the DERF arguments first, sorted into
// the ones its series and its continued fraction evaluate so that a warp runs
// one of the two on full lanes, then (layer, band) items for the band sums,
// and last a lane per level writes every array contiguously (the layer's
// properties, or the routines' defaults).  Bound by the FP64 work of the
// DERFs (80 steps of the continued fraction for half of the 21 edges of a
// layer; issue 43%).  4,050 x 24 columns of dust and ice: 381 -> 181 us
// against going layer by layer across a column's warp -- 21 lanes for the
// edges, both DERF branches in one warp, 12 lanes for the bands, two levels
// written per array.
#include "rt_aerosol.cuh"
#include "../../include/mgcm_rt_math.h"

namespace mgcm {

namespace {

__device__ __forceinline__ double r4(double x) { return (double)(float)x; }

// Size parameters of one layer's lognormal distribution (OPT_DST / OPT_CLD):
// whether the layer passes the routine's thresholds, the core-ratio row of
// the ice tables, 1/Rs and the cross-section factor Ao.
struct LayerMie {
    double rs_inv, ao;
    int irap;
};

template <bool CLD>
__device__ bool layer_mie(const AeroConst &K, double ma, double mcor, double nb, LayerMie &m) {
    const double PIc = 3.1415926535897932;
    const double athird = (double)(1.0f / 3.0f);
    const double dpden_dt = r4(2.5E+3), dpden_ice = r4(917.);
    bool do_it;
    int irap = AERO_NRATIO;
    double Mo = 0.0, No = 0.0, dens = 0.0;
    if (!CLD) {
        do_it = ma > r4(1.e-8) && nb > 1.0;
        Mo = ma;
        No = nb + 1.0;
        dens = dpden_dt;
    } else {
        do_it = ma + mcor > r4(1.e-7) && nb > 1.0;
        if (do_it) {
            float mtc = (float)(mcor / dpden_dt / (ma / dpden_ice + mcor / dpden_dt));
            mtc = (float)mgcm_rt_pow((double)mtc, athird);
            for (int i = 1; i <= AERO_NRATIO; ++i) {
                const float cr = K.cor_ratio[i - 1];
                if (mtc < cr && i != 1) {
                    irap = i - 1;
                    break;
                } else if (mtc == cr) {
                    irap = i;
                    break;
                } else if (mtc < cr && i == 1) {
                    irap = 1;
                    break;
                }
            }
            Mo = ma + mcor;
            No = nb;
            dens = ma / Mo * dpden_ice + mcor / Mo * dpden_dt;
        }
    }
    if (!do_it) return false;
    const double dev = CLD ? r4(0.3087) : r4(0.63676);
    const double cst = 0.75 / (PIc * dens);
    double Rs = mgcm_rt_pow(Mo / No * cst, athird) * mgcm_rt_exp(-0.5 * (dev * dev));
    m.ao = No * PIc * (Rs * Rs);
    Rs = Rs * mgcm_rt_exp(1.5 * (dev * dev));
    Rs = fmin(fmax(Rs, r4(1.e-7)), CLD ? r4(100.e-6) : r4(50.e-6));
    m.rs_inv = 1.0 / Rs;
    m.irap = irap;
    return true;
}

constexpr int AERO_CHUNK = 16;              // layers at a time
constexpr int AERO_EDGES = AERO_NBIN + 1;
constexpr int AERO_BANDS = AERO_NV + AERO_NI;

// One warp's shared memory.
struct AeroWarp {
    LayerMie lm[AERO_CHUNK];
    double e[AERO_CHUNK * AERO_EDGES];              // DERF arguments, values, then bin weights
    double opt[AERO_CHUNK][AERO_BANDS][3];          // QEXT, QSCAT, G per layer and band
    unsigned short item[AERO_CHUNK * AERO_EDGES];   // DERF items: series from the front, fraction from the back
    unsigned char layer[AERO_CHUNK];                // the chunk's layers with aerosol
};

// Layers 16q+1 .. 16q+16 of a column and their levels; with q = 0 also levels
// 1-3 and L_LEVELS+1, which always hold the defaults.
template <bool CLD>
__device__ void layer_chunk(int lane, const AeroConst &K, const double *__restrict__ mie, int L, int q,
                            const double *pl, const double *ma, const double *mcor, const double *nb, AeroWarp &w,
                            double *tauref, double *qextref, double *qxv, double *qsv, double *gv, double *qxi,
                            double *qsi, double *gi) {
    const unsigned full = 0xffffffffu;
    const int lev = 2 * L + 3, lev1 = lev + 1;
    const double GRAVc = 3.72;
    const double dev = CLD ? r4(0.3087) : r4(0.63676);
    const double dev2 = 1.0 / ((double)sqrtf(2.0f) * dev);
    bool on = false;
    const int l = AERO_CHUNK * q + lane + 1;
    if (lane < AERO_CHUNK && l <= L) on = layer_mie<CLD>(K, ma[l - 1], CLD ? mcor[l - 1] : 0.0, nb[l - 1], w.lm[lane]);
    const unsigned mask = __ballot_sync(full, on);
    const unsigned below = (1u << lane) - 1u;
    if (on) w.layer[__popc(mask & below)] = (unsigned char)lane;
    __syncwarp();
    const int non = __popc(mask), nedge = non * AERO_EDGES;
    // DERF arguments, sorted by the branch mgcm_rt_erf takes
    int na = 0, nf = 0;
    for (int i0 = 0; i0 < nedge; i0 += 32) {
        const int i = i0 + lane;
        bool ser = false, frac = false;
        if (i < nedge) {
            const int r = i / AERO_EDGES;
            const double x = mgcm_rt_ln(K.radb[i - r * AERO_EDGES] * w.lm[w.layer[r]].rs_inv) * dev2;
            const double ax = fabs(x);
            ser = ax < 1.5;
            frac = !ser && !(ax >= 6.0);
            w.e[i] = ser || frac ? x : mgcm_rt_erf(x);
        }
        const unsigned ms = __ballot_sync(full, ser), mf = __ballot_sync(full, frac);
        if (ser) w.item[na + __popc(ms & below)] = (unsigned short)i;
        if (frac) w.item[AERO_CHUNK * AERO_EDGES - 1 - nf - __popc(mf & below)] = (unsigned short)i;
        na += __popc(ms);
        nf += __popc(mf);
    }
    __syncwarp();
    for (int i = lane; i < na; i += 32) w.e[w.item[i]] = mgcm_rt_erf(w.e[w.item[i]]);
    for (int i = lane; i < nf; i += 32) {
        const int j = w.item[AERO_CHUNK * AERO_EDGES - 1 - i];
        w.e[j] = mgcm_rt_erf(w.e[j]);
    }
    __syncwarp();
    // bin weights in place of the edges below them
    for (int i0 = 0; i0 < nedge; i0 += 32) {
        const int i = i0 + lane;
        const double s = i + 1 < nedge ? 0.5 * (w.e[i + 1] - w.e[i]) : 0.0;
        __syncwarp();
        if (i < nedge) w.e[i] = s;
        __syncwarp();
    }
    // band sums over the 20 bins in the routine's order (the layer's two
    // levels have the same); mie layout: dust [3][bin][7] vis, [3][bin][5]
    // IR; ice [3][ratio][bin][7], [3][ratio][bin][5]
    for (int i = lane; i < non * AERO_BANDS; i += 32) {
        const int r = i / AERO_BANDS, b = i - r * AERO_BANDS;
        const bool vis = b < AERO_NV;
        const int iw = vis ? b : b - AERO_NV, nbd = vis ? AERO_NV : AERO_NI, ly = w.layer[r];
        const double *tab;
        size_t sq;
        if (vis) {
            tab = CLD ? mie + AERO_DST_SIZE + (size_t)(w.lm[ly].irap - 1) * AERO_NBIN * AERO_NV : mie;
            sq = CLD ? (size_t)AERO_NRATIO * AERO_NBIN * AERO_NV : (size_t)AERO_NBIN * AERO_NV;
        } else {
            tab = CLD ? mie + AERO_DST_SIZE + 3 * AERO_NRATIO * AERO_NBIN * AERO_NV +
                            (size_t)(w.lm[ly].irap - 1) * AERO_NBIN * AERO_NI
                      : mie + 3 * AERO_NBIN * AERO_NV;
            sq = CLD ? (size_t)AERO_NRATIO * AERO_NBIN * AERO_NI : (size_t)AERO_NBIN * AERO_NI;
        }
        double x = 0.0, sc = 0.0, g = 0.0;
        const double *sf = w.e + r * AERO_EDGES;
#pragma unroll 4
        for (int n = 0; n < AERO_NBIN; ++n) {
            const double f = sf[n];
            x = x + f * __ldg(tab + n * nbd + iw);
            sc = sc + f * __ldg(tab + sq + n * nbd + iw);
            g = g + f * __ldg(tab + 2 * sq + n * nbd + iw);
        }
        w.opt[ly][b][0] = x;
        w.opt[ly][b][1] = fmin(sc, r4(0.99999) * x);
        w.opt[ly][b][2] = g;
    }
    __syncwarp();
    auto level = [&](int k, int ly, bool act) {
        const double q6 = act ? w.opt[ly][5][0] : 1.0;   // QXV of L_NREFV = 6
        qextref[k - 1] = q6;
        tauref[k - 1] = act ? w.lm[ly].ao * q6 * (100.0 * (pl[k - 1] - pl[k - 2]) / GRAVc) : 0.0;
        for (int b = 0; b < AERO_BANDS; ++b) {
            const bool vis = b < AERO_NV;
            const int o = (vis ? b : b - AERO_NV) * lev1 + k - 1;
            (vis ? qxv : qxi)[o] = act ? w.opt[ly][b][0] : 1.0;
            (vis ? qsv : qsi)[o] = act ? w.opt[ly][b][1] : 1.0 * r4(0.99);
            (vis ? gv : gi)[o] = act ? w.opt[ly][b][2] : 0.0;
        }
    };
    const int k = 4 + 2 * AERO_CHUNK * q + lane, ly = lane >> 1;
    if (k <= lev) level(k, ly, (mask >> ly) & 1u);
    if (q == 0 && lane < 4) level(lane < 3 ? lane + 1 : lev1, 0, false);
    __syncwarp();   // the shared arrays are rewritten by the next chunk
}

}  // namespace

__global__ void __launch_bounds__(32 * AERO_WARPS, 6)
rt_aerosol(const AeroSeg a, const __grid_constant__ AeroConst K, const double *__restrict__ mie) {
    __shared__ AeroWarp ws[AERO_WARPS];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int L = a.L, lev = 2 * L + 3, lev1 = lev + 1;
    // a warp's task is one chunk of one family of a column, the dust (more
    // layers) first
    const int nq = (L + AERO_CHUNK - 1) / AERO_CHUNK;
    const long long per = (long long)a.ncol * nq, tasks = per * (a.active_dust + a.cloudon);   // prescribed dust: none
    for (long long i = (long long)blockIdx.x * AERO_WARPS + wid; i < tasks; i += (long long)gridDim.x * AERO_WARPS) {
        const long long j = i % per;
        const size_t c = (size_t)(j / nq);
        const int q = (int)(j % nq);
        const double *pl = a.plev + c * lev;
        if (a.active_dust && i < per)
            layer_chunk<false>(lane, K, mie, L, q, pl, a.dust_mass + c * L, nullptr, a.dust_number + c * L, ws[wid],
                               a.tauref + c * lev1, a.qextrefdst + c * lev1, a.qxvdst + c * AERO_NV * lev1,
                               a.qsvdst + c * AERO_NV * lev1, a.gvdst + c * AERO_NV * lev1,
                               a.qxidst + c * AERO_NI * lev1, a.qsidst + c * AERO_NI * lev1,
                               a.gidst + c * AERO_NI * lev1);
        else
            layer_chunk<true>(lane, K, mie, L, q, pl, a.ice_mass + c * L, a.ice_core + c * L, a.ice_number + c * L,
                              ws[wid], a.taurefcld + c * lev1, a.qextrefcld + c * lev1, a.qxvcld + c * AERO_NV * lev1,
                              a.qsvcld + c * AERO_NV * lev1, a.gvcld + c * AERO_NV * lev1, a.qxicld + c * AERO_NI * lev1,
                              a.qsicld + c * AERO_NI * lev1, a.gicld + c * AERO_NI * lev1);
    }
}

}  // namespace mgcm

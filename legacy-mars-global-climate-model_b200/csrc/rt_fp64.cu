// Plain FP64 column radiative transfer, reference operation order.
//
// One CTA per column (persistent grid-stride loop over the columns of every
// segment), 224 threads: thread s < 119 owns visible system (nw, ng) =
// (s/17+1, s%17+1), 119 <= s < 204 owns IR system ((s-119)/17+1, ...).
//
// Per system the reference calls OPTCV/OPTCI (one column of DTAUK),
// GETDETAU, then GFLUXV/GFLUXI -> DSOLVER -> DTRIDGL.  Here a system runs:
//   pass A  top-down over levels: 8-corner k gather and H2O/T/P interpolation
//           (code/optcv.f90:128-176, code/optci.f90:143-167), cumulative TAUCUM,
//           per-layer DTAU/WBAR and the delta-Eddington scaling
//           (code/getdetau.f90:29-56 = code/gfluxv.f90:76-103);
//   pass C  bottom-up over layers: two-stream coefficients
//           (code/gfluxv.f90:108-163, code/gfluxi.f90:69-123), the DSOLVER rows
//           (code/dsolver.f90:54-85) generated in the order DTRIDGL eliminates
//           them (code/dtridgl.f90:25-32), eliminated on the fly;
//   pass D  top-down: DTRIDGL back-substitution (code/dtridgl.f90:34-38),
//           unmixing (code/dsolver.f90:91-103) and the midpoint fluxes
//           (code/gfluxv.f90:170-280, code/gfluxi.f90:136-194).
// The flux sums over bands and Gauss points are then formed by one thread
// per output in the reference's order (code/sfluxv.f90:60-164,
// code/sfluxi.f90:57-145) and turned into SUNTOT/IRTOTAL/QRAD
// (code/comp3.f:677-681,735-738,765-771).
//
// Built with --fmad=false: like the reference's x86-64 build, no multiply-add
// is contracted, so every operation rounds as the Fortran does.  Every
// exponential goes through mgcm_rt_exp (include/mgcm_rt_math.h), the routine
// the CPU oracle uses too, so host and device agree bit-for-bit.
#include "rt_fp64_sys.cuh"
#include "rt_quad.cuh"
#include "rt_solve.cuh"
#include "../../include/mgcm_rt_math.h"

namespace mgcm {

using namespace fp64;

__global__ void __launch_bounds__(224, 2)
rt_fp64_kernel(const SegTable *__restrict__ st, const double *__restrict__ kv,
               const double *__restrict__ ki, const double *__restrict__ planck,
               const RtConst K, int max_nl, uint32_t *status, unsigned long long *nsys,
               double *red_scratch) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ColSmem s = carve_smem(smem_raw, max_nl,
                           red_scratch ? red_scratch + (size_t)blockIdx.x * 2 * NSYS * max_nl : nullptr);
    SysLocal w;
    unsigned int nsolved = 0;
    const int total = st->total_cols;
    for (int g = blockIdx.x; g < total; g += gridDim.x) {
        const int si = find_seg(st, g);
        const SegDev &sg = st->seg[si];
        const int c = g - sg.col0;
        const int L = sg.L, NL = L + 1, LEV = 2 * L + 3;
        const bool day = sg.acosz[c] >= R4(1.0e-5);
        stage_column(sg, c, K, planck, s, status);
        __syncthreads();
        const int t = threadIdx.x;
        if (t < NSYS_V) {
            if (day)
                solve_vis<0>(sg, c, t / D_NG + 1, t % D_NG + 1, t, s, K, kv, w, nsolved,
                             s.fmp + (size_t)t * NL, s.fmm + (size_t)t * NL, &s.sc0[t], &s.sc1[t],
                             &s.sc2[t]);
        } else if (t < NSYS) {
            const int j = t - NSYS_V;
            solve_ir<0>(sg, c, j / D_NG + 1, j % D_NG + 1, t, s, K, ki, w, nsolved,
                        s.fmp + (size_t)t * NL, s.fmm + (size_t)t * NL, &s.sc0[t]);
        }
        __syncthreads();
        reduce_and_heat(
            sg, c, [&](bool vis, int q, int l) { return reduce_family(s, K, vis, q, l, NL); },
            s.fmnet_v, s.fmnet_i, s.misc, day);
        __syncthreads();
    }
    if (nsys) {
        // warp-aggregated count of solved systems
        unsigned int v = nsolved;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0 && v) atomicAdd(nsys, (unsigned long long)v);
    }
}

// ---------------------------------------------------------------------------
// Three-kernel pipeline over a chunk of columns [col_begin, col_end).  Each
// column owns a block of global memory laid out like the fused kernel's shared
// memory (ColSmem, stride bytes): the stage data, the TLIMIT flags and the
// per-system midpoint fluxes.  Solved systems are listed per family so the
// solver keeps every thread busy (night columns and TLIMIT skips drop out).

// K0: stage the columns (bins, per-band opacity terms, Planck terms) into
// their global blocks, `cols` (1..STAGE_COLS) columns per CTA at a time: the
// level items of all of them, a barrier, then a warp per (column, band), its
// lanes along the layers.  The TAUREF ratios live in shared memory between
// the two.  8,192 x 24 columns: 200 -> 156 us against items in (layer, band)
// order, whose lanes read 54 values apart and wrote single values of records
// 48 and 64 bytes apart; with the solves' records now contiguous the 64,800 x
// 24 call takes 9.27 -> 8.98 ms.
constexpr int STAGE_COLS = 4;

template <bool V>   // V: check the inputs (Check, rt_stage.cuh)
__global__ void __launch_bounds__(256, 4)   // 64 registers
rt_stage(const SegTable *__restrict__ st, int col_begin, int col_end, int max_nl,
         unsigned char *__restrict__ blocks, size_t stride, const double *__restrict__ planck,
         const __grid_constant__ RtConst K, uint32_t *status, int cols) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int lev1 = 2 * max_nl + 3;   // levels up to LEV+1 = 2NL+2, 1-based
    double *tref = reinterpret_cast<double *>(smem_raw);
    auto column = [&](int g, int j) {
        ColSmem s = carve_smem(blocks + (size_t)(g - col_begin) * stride, max_nl, nullptr, false);
        s.tref_v = tref + (3 * j) * lev1;
        s.tref_i = tref + (3 * j + 1) * lev1;
        s.tref_c = tref + (3 * j + 2) * lev1;
        return s;
    };
    for (int g0 = col_begin + blockIdx.x * cols; g0 < col_end; g0 += gridDim.x * cols) {
        const int ng = min(cols, col_end - g0);
        for (int j = 0; j < ng; ++j) {
            const SegDev &sg = st->seg[find_seg(st, g0 + j)];
            ColSmem s = column(g0 + j, j);
            // the columns' items follow one another over the CTA's threads
            const int per = 2 * sg.L + 3, t = (int)(threadIdx.x + blockDim.x - (j * 64) % blockDim.x) % (int)blockDim.x;
            for (int it = t; it < per; it += blockDim.x) stage_level<V>(sg, g0 + j - sg.col0, K, s, 2 + it, status);
        }
        __syncthreads();
        for (int u = wid; u < ng * (D_NV + D_NI); u += nw) {
            const int j = u / (D_NV + D_NI), b = u - j * (D_NV + D_NI);
            const SegDev &sg = st->seg[find_seg(st, g0 + j)];
            ColSmem s = column(g0 + j, j);
            for (int l = lane; l <= sg.L + 1; l += 32) stage_band<V>(sg, g0 + j - sg.col0, K, planck, s, b, l, status);
        }
        __syncthreads();
    }
}
size_t stage_smem_bytes(int max_nl) { return (size_t)STAGE_COLS * 3 * (2 * max_nl + 3) * sizeof(double); }

#define STAGE_ARGS                                                                                     \
    const SegTable *__restrict__, int, int, int, unsigned char *__restrict__, size_t,                \
        const double *__restrict__, const __grid_constant__ RtConst, uint32_t *, int
template __global__ void rt_stage<false>(STAGE_ARGS);
template __global__ void rt_stage<true>(STAGE_ARGS);
#undef STAGE_ARGS

// K1: screen every system (optics sums, TLIMIT test, DETAU, CUMTAUV) and
// append the kept ones to the family lists.  F32 (mixed precision): visible
// gas opacities from the FP32 table; the IR family always screens in FP64.
// One warp per (column, group); warps never wait on one another.  `groups` is
// SCREEN_GROUPS_V when the solve screens the IR systems itself (rt_ir_dense).  A group's kept systems take one
// contiguous run of list positions in ascending order; its base and count go
// to the column's meta words.
template <bool F32>
__global__ void __launch_bounds__(128, 8)   // 64 registers (5 / 6 / 8 CTAs per SM: 10.60 / 10.45 / 10.34 ms)
rt_fp64_screen(const SegTable *__restrict__ st, int col_begin, int col_end, int max_nl,
               unsigned char *__restrict__ blocks, size_t stride, const double *__restrict__ kv,
               const double *__restrict__ ki, const __grid_constant__ RtConst K, int *__restrict__ list_v,
               int *__restrict__ list_i, unsigned int *counts, unsigned long long *nsys,
               const float *__restrict__ kvf, int groups) {
    SolveLocal w;
    unsigned int nsolved = 0;
    const int lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const int items = (col_end - col_begin) * groups;
    for (int it = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; it < items; it += nwarps) {
        const int g = col_begin + it / groups, grp = it % groups;
        const SegDev &sg = st->seg[find_seg(st, g)];
        const int c = g - sg.col0;
        unsigned char *block = blocks + (size_t)(g - col_begin) * stride;
        ColSmem s = carve_smem(block, max_nl, nullptr, false);
        const bool vis = grp < SCREEN_GROUPS_V;
        const int t = group_first(grp) + lane;
        bool act = false;
        if (vis) {
            if (t < group_end(grp) && sg.acosz[c] >= R4(1.0e-5))
                act = fast_vis_screen<F32>(sg, c, t, block, max_nl, s, K, kv, kvf, w, nsolved);
        } else if (t < group_end(grp)) {
            const int j = t - NSYS_V;
            solve_ir<1>(sg, c, j / D_NG + 1, j % D_NG + 1, t, s, K, ki, w.g, nsolved, nullptr, nullptr,
                        nullptr);
            act = s.skip[t] == 0;
        }
        const unsigned m = __ballot_sync(0xffffffffu, act);
        const int n = __popc(m);
        int base = 0;
        if (lane == 0) {
            base = n ? (int)atomicAdd(&counts[vis ? 0 : 1], (unsigned)n) : 0;
            s.meta[2 * grp] = base;
            s.meta[2 * grp + 1] = n;
        }
        base = __shfl_sync(0xffffffffu, base, 0);
        if (act) (vis ? list_v : list_i)[base + __popc(m & ((1u << lane) - 1u))] = (g << 8) | t;
    }
    if (nsys) {
        unsigned int v = nsolved;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0 && v) atomicAdd(nsys, (unsigned long long)v);
    }
}

#define SCREEN_ARGS                                                                                    \
    const SegTable *__restrict__, int, int, int, unsigned char *__restrict__, size_t,                \
        const double *__restrict__, const double *__restrict__, const __grid_constant__ RtConst, int *__restrict__,    \
        int *__restrict__, unsigned int *, unsigned long long *, const float *__restrict__, int
template __global__ void rt_fp64_screen<false>(SCREEN_ARGS);
template __global__ void rt_fp64_screen<true>(SCREEN_ARGS);
#undef SCREEN_ARGS

// K2: solve the listed visible systems, one thread per system.
__global__ void __launch_bounds__(128, MGCM_VIS_SOLVE_MINB)
rt_fp64_solve_vis(const SegTable *__restrict__ st, int col_begin, int max_nl,
                  unsigned char *__restrict__ blocks, size_t stride, const double *__restrict__ ktab,
                  const __grid_constant__ RtConst K, const int *__restrict__ list, const unsigned int *count,
                  double *__restrict__ fl, double *__restrict__ sc) {
    SolveLocal w;
    const unsigned int n = count[0];
    for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int e = list[i];
        const int g = e >> 8;
        const SegDev &sg = st->seg[find_seg(st, g)];
        double *row = fl + row_base(i, max_nl);
        fast_vis<false>(sg, g - sg.col0, e & 255, blocks + (size_t)(g - col_begin) * stride, max_nl, K, ktab,
                        nullptr, w, row, row + (size_t)max_nl * ROW_BLK, sc + sc_base(i));
    }
}

// K1 and K2 in one for small calls: screen and solve the visible systems of a
// chunk, one thread per system, at list position (column) * 119 + system.
// Half of a day column's systems pass the screen, so most warps carry idle
// lanes through the solve; but where all of them are resident at once that
// costs nothing, and the call is spared a kernel and a second pass A in its
// longest chain of dependent kernels.  FP64 only: MIXED solves contract
// multiply-adds (rt_mixed.cu), and a column's result must not depend on the
// size of the call.  60 / 200 / 400 x 24 columns: 191 / 198 / 229 -> 163 / 179 /
// 220 us; 800: 269 -> 311, so three columns per SM is the limit.
__global__ void __launch_bounds__(128, MGCM_VIS_SOLVE_MINB)
rt_vis_dense(const SegTable *__restrict__ st, int col_begin, int col_end, int max_nl,
             unsigned char *__restrict__ blocks, size_t stride, const double *__restrict__ kv,
             const __grid_constant__ RtConst K, double *__restrict__ fl,
             double *__restrict__ sc, unsigned long long *nsys) {
    SolveLocal w;
    unsigned int nsolved = 0;
    const int n = (col_end - col_begin) * NSYS_V;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int cc = i / NSYS_V, g = col_begin + cc;
        const SegDev &sg = st->seg[find_seg(st, g)];
        const int c = g - sg.col0;
        if (!(sg.acosz[c] >= R4(1.0e-5))) continue;
        double *row = fl + row_base(i, max_nl);
        nsolved += fast_vis<false, true>(sg, c, i - cc * NSYS_V, blocks + (size_t)cc * stride, max_nl, K, kv, nullptr, w, row,
                                       row + (size_t)max_nl * ROW_BLK, sc + sc_base(i));
    }
    if (nsys) {
        for (int o = 16; o > 0; o >>= 1) nsolved += __shfl_down_sync(0xffffffffu, nsolved, o);
        if ((threadIdx.x & 31) == 0 && nsolved) atomicAdd(nsys, (unsigned long long)nsolved);
    }
}

// K2: screen and solve the IR systems of a chunk, one thread per system, at
// list position (column in the chunk) * 85 + system.  Nine tenths of them
// pass TLIMIT, so a list of the kept ones would fill 8% more lanes but take
// every gas optical depth twice, in a screen and here; the threads of a
// screened system wait.  With the fast arithmetic (rt_solve.cuh) the call
// of 64,800 x 24 columns takes 13.4 -> 11.45 ms (FP64), the screen of 8,192
// columns 433 -> 365 us, both solves 1,185 -> 1,090 us.
__global__ void __launch_bounds__(128, MGCM_IR_SOLVE_MINB)
rt_ir_dense(const SegTable *__restrict__ st, int col_begin, int col_end, int max_nl,
            unsigned char *__restrict__ blocks, size_t stride, const double *__restrict__ ktab,
            const __grid_constant__ RtConst K, double *__restrict__ fl, double *__restrict__ sc,
            unsigned long long *nsys) {
    SolveLocal w;
    unsigned int nsolved = 0;
    const int n = (col_end - col_begin) * NSYS_I;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        nsolved += fast_ir(st, col_begin, i, max_nl, blocks, stride, K, ktab, w, fl, sc) == 0;
    }
    if (nsys) {
        for (int o = 16; o > 0; o >>= 1) nsolved += __shfl_down_sync(0xffffffffu, nsolved, o);
        if ((threadIdx.x & 31) == 0 && nsolved) atomicAdd(nsys, (unsigned long long)nsolved);
    }
}

// K2 (four-lane form, L <= 51): a quad of lanes per kept system, 8 systems
// per warp, per-layer values in registers (rt_quad.cuh).  A quad past the
// end of the list repeats the last system and stores nothing.
template <bool VIS, int R>
__global__ void __launch_bounds__(128)
rt_quad_solve(const SegTable *__restrict__ st, int col_begin, int max_nl,
              unsigned char *__restrict__ blocks, size_t stride, const double *__restrict__ ktab,
              const RtConst K, const int *__restrict__ list, const unsigned int *count,
              double *__restrict__ fl, double *__restrict__ sc) {
    const unsigned int n = VIS ? count[0] : count[1];
    const unsigned int lane = threadIdx.x & 31;
    const unsigned int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (unsigned int base = warp * 8; base < n; base += nwarps * 8) {
        const unsigned int i = base + (lane >> 2);
        const bool live = i < n;
        const unsigned int ii = live ? i : n - 1;
        const int e = list[ii];
        const int g = e >> 8, sidx = e & 255;
        const SegDev &sg = st->seg[find_seg(st, g)];
        const int c = g - sg.col0;
        const ColSmem s = carve_smem(blocks + (size_t)(g - col_begin) * stride, max_nl, nullptr, false);
        double *row = fl + row_base(ii, max_nl), *scr = sc + sc_base(ii);
        double *rdn = row + (size_t)max_nl * ROW_BLK;   // downward fluxes
        if (VIS) {
            quad_vis<R, false>(sg, c, sidx / D_NG + 1, sidx % D_NG + 1, s, K, ktab, nullptr, live, row,
                               rdn, scr, ROW_BLK);
        } else {
            const int j = sidx - NSYS_V;
            quad_ir<R>(sg, c, j / D_NG + 1, j % D_NG + 1, s, K, ktab, live, row, rdn, scr,
                       ROW_BLK);
        }
    }
}

#define QUAD_ARGS                                                                                      \
    const SegTable *__restrict__, int, int, unsigned char *__restrict__, size_t, const double *__restrict__, \
        const RtConst, const int *__restrict__, const unsigned int *, double *__restrict__,             \
        double *__restrict__
template __global__ void rt_quad_solve<true, 7>(QUAD_ARGS);
template __global__ void rt_quad_solve<true, 10>(QUAD_ARGS);
template __global__ void rt_quad_solve<true, 13>(QUAD_ARGS);
template __global__ void rt_quad_solve<false, 7>(QUAD_ARGS);
template __global__ void rt_quad_solve<false, 10>(QUAD_ARGS);
template __global__ void rt_quad_solve<false, 13>(QUAD_ARGS);
#undef QUAD_ARGS

// K3: ordered sums and heating, one warp per column.  The solves store their
// flux rows in blocks of 32 list positions (row_base, sc_base): value k of
// the system at position p is fl[row_base(p) + 32 k] (k < max_nl: upward
// midpoint flux of layer k+1; max_nl + k: downward), scalar q
// sc[sc_base(p) + 32 q].  A column's kept systems sit in ascending (band,
// Gauss) order, in one run of positions per screening group or, per `dense`,
// at 119 (DENSE_V, rt_vis_dense) and 85 (DENSE_I, rt_ir_dense) positions a column.
//
// The rows of up to 16 systems at a time come into shared memory with
// asynchronous copies, half a warp along the systems for the upward and half
// for the downward fluxes (a value of 16 consecutive positions is one
// 128-byte segment), at a pitch of 17; then a lane per
// level sums its outputs over the systems in the reference order, reading
// the buffer without bank conflicts.  8,192 x 24 columns: 255 -> 191 us against
// loading the rows lane by level straight from global memory, 32 cache lines
// a value, which ran at 76% of the L1's tag rate; what bounds it now is the
// latency of its short phases at 8 warps per SM (the carve-out set beside its
// attributes; issue 29%, 2.4 TB/s).  32 systems at a time: the same at 24
// layers, 1.5% slower calls at 48.
constexpr int RED_LPL = (D_MAXNL + 2 + 31) / 32;   // items (levels and two scalar sums) per lane
constexpr int RED_SYS = 16, RED_PITCH = RED_SYS + 1;   // systems staged at a time

// A kept system: its multipliers m1, m2, m3 as family_multipliers gives them,
// its list position, and which factors are not exactly 1.0 (bit 0: m2, bit 1: m3).
struct alignas(16) RedSys {
    double a, b, e;
    int pos, fac;
};

// Shared memory of a CTA: FMNET per level of both families, the two factors
// of the heating rate and the top values; then per warp one family's kept
// systems and the staged rows: NL + 2 items, upward and downward.
__host__ __device__ inline size_t red_col_bytes(int max_nl) {
    return ((size_t)(4 * (max_nl + 1) + 2) * 8 + 15) / 16 * 16;
}
__host__ __device__ inline size_t red_warp_bytes(int max_nl) {
    return (size_t)NSYS_V * sizeof(RedSys) + (size_t)2 * (max_nl + 2) * RED_PITCH * 8;
}

// Multipliers of one family of a column, one lane per band: `mine` holds, on
// lane w, the kept flags of systems 32w .. 32w+31 of the family.  Each lane
// walks its band as family_multipliers does, at the band's offset among the
// kept rows.
__device__ inline void warp_multipliers(unsigned mine, bool vis, const RtConst &K, RedSys *sys) {
    const int lane = threadIdx.x & 31;
    const bool on = lane < (vis ? D_NV : D_NI);
    const double fz = on ? (vis ? K.fzerov[lane] : K.fzeroi[lane]) : 0.0;
    const int first = (on ? lane : 0) * D_NG, w = first >> 5;
    const unsigned lo = __shfl_sync(0xffffffffu, mine, w), hi = __shfl_sync(0xffffffffu, mine, w + 1);
    const unsigned bits = __funnelshift_r(lo, hi, first & 31) & 0xffffu;   // points 1..16
    const bool gas = !(fz >= R4(0.99));
    const int cnt = on ? (gas ? __popc(bits) : 0) + 1 : 0;
    int pos = cnt;   // exclusive prefix over the bands
    for (int o = 1; o < 8; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, pos, o);
        if (lane >= o) pos += v;
    }
    pos -= cnt;
    if (!on) return;
    double fzero = fz;
    const double dw = vis ? 1.0 : K.dwni[lane], one = 1.0 - fz;
    auto put = [&](double a, double b, double e) {
        RedSys &r = sys[pos++];
        r.a = a;
        r.b = b;
        r.e = e;
        r.fac = (b != 1.0 ? 1 : 0) | (e != 1.0 ? 2 : 0);
    };
    if (gas) {
        for (int ng = 0; ng < D_NG - 1; ++ng) {
            if (!((bits >> ng) & 1u)) fzero = fzero + one * K.gweight[ng];
            else if (vis) put(K.gweight[ng], one, 1.0);
            else put(dw, K.gweight[ng], one);
        }
    }
    if (vis) put(fzero, 1.0, 1.0);
    else put(dw, fzero, 1.0);
}

// 8 bytes from global to shared memory, asynchronously.
__device__ __forceinline__ void copy8_async(double *dst, const double *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}

template <int RB>   // systems whose staged values are read before they are summed
__global__ void __launch_bounds__(64)
rt_fp64_reduce(const SegTable *__restrict__ st, int col_begin, int col_end, int max_nl,
               unsigned char *__restrict__ blocks, size_t stride, const __grid_constant__ RtConst K,
               const double *__restrict__ fl_v, const double *__restrict__ sc_v,
               const double *__restrict__ fl_i, const double *__restrict__ sc_i, int dense) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // one warp per column, or two with a family each (small calls)
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const bool two = blockDim.x > 32;
    double *fmv = reinterpret_cast<double *>(smem_raw), *fmi = fmv + max_nl + 1;   // [1..NL]
    double *pnl = fmi + max_nl + 1, *den = pnl + max_nl + 1, *misc = den + max_nl + 1;
    RedSys *sys = reinterpret_cast<RedSys *>(smem_raw + red_col_bytes(max_nl) + wid * red_warp_bytes(max_nl));
    double *buf = reinterpret_cast<double *>(sys + NSYS_V);

    for (int g = col_begin + blockIdx.x; g < col_end; g += gridDim.x) {
        const SegDev &sg = st->seg[find_seg(st, g)];
        const int c = g - sg.col0;
        const int NL = sg.L + 1, LEV = 2 * NL + 1, R = NL + 2;   // staged items: the levels, FLUXUP/FLUXDN at the top, DIFFV
        const ColSmem s = carve_smem(blocks + (size_t)(g - col_begin) * stride, max_nl, nullptr, false);
        const bool day = sg.acosz[c] >= R4(1.0e-5);
        // kept flags of both families: lane w holds those of systems 32w .. 32w+31
        unsigned mine_v = 0, mine_i = 0;
        {
            unsigned char f[7];
#pragma unroll
            for (int w = 0; w < 7; ++w) {
                const int t = w < 4 ? 32 * w + lane : NSYS_V + 32 * (w - 4) + lane;
                f[w] = t < (w < 4 ? NSYS_V : NSYS) ? s.skip[t] : 1;
            }
#pragma unroll
            for (int w = 0; w < 7; ++w) {
                const unsigned m = __ballot_sync(0xffffffffu, f[w] == 0);
                if (w < 4 && lane == w) mine_v = m;
                if (w >= 4 && lane == w - 4) mine_i = m;
            }
        }
        if (!day) mine_v = 0;
        const int gbase = lane < SCREEN_GROUPS ? s.meta[2 * lane] : 0;   // list positions of the groups
        // what the heating rates need besides the fluxes (code/comp3.f:765-771)
        const double *plev = sg.plev + (size_t)c * LEV;
        for (int l = 1 + threadIdx.x; l <= NL; l += blockDim.x) {
            const int k = 2 * l;
            const double ptrop = sg.ptrop;
            const double ym = k == 2 ? ptrop * 100.0 / 3.72 : (plev[k + 1 - 1] - plev[k - 1 - 1]) * 100.0 / 3.72;
            const double om = pow(plev[k - 1] / plev[LEV - 1], 0.25684);
            pnl[l] = sg.sigma[k - 1] * (sg.pcol[c] - ptrop) + ptrop;
            den[l] = 735.94 * ym * om;
        }
        for (int fam = two ? wid : 0; fam < (two ? wid + 1 : 2); ++fam) {
            const bool vis = fam == 0;
            const unsigned mine = vis ? mine_v : mine_i;
            // the family's kept systems in order (none at night for the
            // visible family: its outputs are zeros)
            int nrow = 0;
            if (!vis || day) {
                for (int w = 0; w < (vis ? 4 : 3); ++w) {
                    const unsigned m = __shfl_sync(0xffffffffu, mine, w);
                    const int base = __shfl_sync(0xffffffffu, gbase, vis ? w : 4 + w);
                    const int before = __popc(m & ((1u << lane) - 1u));
                    if ((m >> lane) & 1u)
                        sys[nrow + before].pos = dense & (vis ? DENSE_V : DENSE_I)
                                                     ? (g - col_begin) * (vis ? NSYS_V : NSYS_I) + 32 * w + lane
                                                     : base + before;
                    nrow += __popc(m);
                }
                warp_multipliers(mine, vis, K, sys);
            }
            __syncwarp();
            const double *fl = vis ? fl_v : fl_i, *sc = vis ? sc_v : sc_i;
            double acc[RED_LPL][3];
#pragma unroll
            for (int r = 0; r < RED_LPL; ++r) acc[r][0] = acc[r][1] = acc[r][2] = 0.0;
            for (int f0 = 0; f0 < nrow; f0 += RED_SYS) {
                const int n = min(RED_SYS, nrow - f0), q = lane % RED_SYS;
                const bool down = lane >= RED_SYS;
                if (q < n) {
                    const int p = sys[f0 + q].pos;
                    const double *pr = fl + row_base(p, max_nl) + (down ? (size_t)max_nl * ROW_BLK : 0);
                    const double *ps = sc + sc_base(p);
                    double *bw = buf + q + (down ? R * RED_PITCH : 0);
                    for (int k = 0; k < NL; ++k) copy8_async(bw + k * RED_PITCH, pr + k * ROW_BLK);
                    // FLUXUP and, visible, FLUXDN at the top; DIFFV
                    if (!down || vis) copy8_async(bw + NL * RED_PITCH, down ? ps + ROW_BLK : ps);
                    else bw[NL * RED_PITCH] = 0.0;
                    if (!down && vis) copy8_async(bw + (NL + 1) * RED_PITCH, ps + 2 * ROW_BLK);
                    else bw[(NL + 1) * RED_PITCH] = 0.0;
                }
                asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
                __syncwarp();
#pragma unroll
                for (int r = 0; r < RED_LPL; ++r) {
                    if (32 * r >= R) break;
                    const int it = min(lane + 32 * r, R - 1);
                    const double *bu = buf + it * RED_PITCH, *bd = bu + R * RED_PITCH;
#pragma unroll 1
                    for (int q0 = 0; q0 < n; q0 += RB) {
                        double up[RB], dn[RB];
#pragma unroll
                        for (int q = 0; q < RB; ++q) {   // past n: within the buffer's pitch, not summed
                            up[q] = bu[q0 + q];
                            dn[q] = bd[q0 + q];
                        }
#pragma unroll
                        for (int q = 0; q < RB; ++q) {
                            if (q0 + q < n) {
                                const RedSys y = sys[f0 + q0 + q];
                                // ((v*a)*b)*e in the reference order; a factor that is
                                // exactly 1.0 leaves the product unchanged and is
                                // skipped (warp-uniform)
                                auto wt = [&](double v) {
                                    double x = v * y.a;
                                    if (y.fac & 1) x = x * y.b;
                                    if (y.fac & 2) x = x * y.e;
                                    return x;
                                };
                                acc[r][0] = acc[r][0] + wt(up[q] - dn[q]);
                                acc[r][1] = acc[r][1] + wt(up[q]);
                                acc[r][2] = acc[r][2] + wt(dn[q]);
                            }
                        }
                    }
                }
                __syncwarp();   // the buffer is refilled
            }
#pragma unroll
            for (int r = 0; r < RED_LPL; ++r) {
                const int it = lane + 32 * r, l = it + 1;
                const double a0 = acc[r][0], a1 = acc[r][1], a2 = acc[r][2];
                const size_t o = (size_t)c * NL + it;
                if (it < NL) {
                    if (vis) {
                        sg.fmnetv[o] = a0;
                        sg.fluxupv[o] = a1;
                        sg.fluxdnv[o] = a2;
                        fmv[l] = a0;
                        if (l == NL) {
                            sg.dnvflux[c] = a2;
                            sg.fluxsurf[c] = (1.0 - sg.als[c]) * a2;
                        }
                    } else {
                        sg.fmneti[o] = a0;
                        sg.fluxupi[o] = a1;
                        sg.fluxdni[o] = a2;
                        fmi[l] = a0;
                        if (l == NL) sg.dnirflux[c] = a2;
                    }
                } else if (it == NL) {
                    (vis ? sg.nfluxtopv : sg.nfluxtopi)[c] = a0;
                    misc[vis ? 0 : 1] = a0;
                } else if (it == NL + 1 && vis) {
                    sg.diffvt[c] = a1;
                    sg.dndiffv[c] = a1;
                }
            }
            __syncwarp();   // sys is rewritten by the next family
        }
        // divergences and heating rates (code/comp3.f:677-681,735-738,765-771)
        if (two) __syncthreads();
        for (int l = 1 + threadIdx.x; l <= NL; l += blockDim.x) {
            const double sun = day ? (l == 1 ? fmv[1] - misc[0] : fmv[l] - fmv[l - 1]) : 0.0;
            const double irt = l == 1 ? fmi[1] - misc[1] : fmi[l] - fmi[l - 1];
            const double sunlte = sun * 2.2e4 * pnl[l] / (1.0 + 2.2e4 * pnl[l]);
            const size_t o = (size_t)c * NL + l - 1;
            sg.suntot[o] = sun;
            sg.irtotal[o] = irt;
            sg.qrad[o] = (sunlte + irt) / den[l];
        }
        // the shared arrays are rewritten by the next column
        if (two) __syncthreads();
        else __syncwarp();
    }
}

#define REDUCE_ARGS                                                                                    \
    const SegTable *__restrict__, int, int, int, unsigned char *__restrict__, size_t,                 \
        const __grid_constant__ RtConst, const double *__restrict__, const double *__restrict__,      \
        const double *__restrict__, const double *__restrict__, int
template __global__ void rt_fp64_reduce<1>(REDUCE_ARGS);
template __global__ void rt_fp64_reduce<2>(REDUCE_ARGS);
template __global__ void rt_fp64_reduce<4>(REDUCE_ARGS);
template __global__ void rt_fp64_reduce<8>(REDUCE_ARGS);
#undef REDUCE_ARGS

// Shared memory of a reduce CTA of `warps` warps.
size_t reduce_smem_bytes(int max_nl, int warps) { return red_col_bytes(max_nl) + warps * red_warp_bytes(max_nl); }
// Systems whose staged values a lane reads before it sums them, by default.
int reduce_rows_per_chunk() { return 4; }
// The reduce kernel of a launch, rb in {1, 2, 4, 8} (other values round down).
const void *reduce_kernel(int rb) {
    if (rb >= 8) return (const void *)rt_fp64_reduce<8>;
    if (rb >= 4) return (const void *)rt_fp64_reduce<4>;
    if (rb >= 2) return (const void *)rt_fp64_reduce<2>;
    return (const void *)rt_fp64_reduce<1>;
}

// Partial radiation: DIRECTSOL from DETAU (code/dsolflux.f:28-45) and
// DNVFLUX = DNDIFFV + DIRECTSOL (code/comp3.f:335-351).
//
// A CTA takes 32 columns: its threads read the columns' DETAU coalesced and
// put the 119 terms of each into shared memory, then a thread per column
// adds them in the reference's order (band by band; a term of DETAU > 5
// counts as +0).  Night columns are not read.
static_assert(NSYS_V <= 128, "a thread per element sets up the tables");
constexpr int DSOL_COLS = 32, DSOL_THREADS = 128, DSOL_ROW = NSYS_V + 2;   // odd pitch: no bank conflicts
constexpr int DSOL_MLP = 8;   // DETAU values a thread has in flight

__global__ void __launch_bounds__(DSOL_THREADS)
rt_dsolflux_kernel(int ncol, const double *__restrict__ sol, const double *__restrict__ acosz,
                   const double *__restrict__ detau, const double *__restrict__ dndiffv,
                   double *__restrict__ dnvflux, const RtConst K) {
    __shared__ double term[DSOL_COLS * DSOL_ROW], u0s[DSOL_COLS], rcp[DSOL_COLS];
    __shared__ int day[DSOL_COLS], nday;   // the tile's day columns
    // per element of DETAU's (Gauss, band) order: SOL, the two weights in the
    // reference's order, and the place in the summation order
    __shared__ double sl[NSYS_V], wa[NSYS_V], wb[NSYS_V];
    __shared__ int at[NSYS_V];
    const int t = threadIdx.x, c0 = blockIdx.x * DSOL_COLS, nc = min(DSOL_COLS, ncol - c0);
    if (t < 32) {
        const double u0 = t < nc ? acosz[c0 + t] : 0.0;
        const bool on = u0 >= R4(1.0e-5);
        const unsigned m = __ballot_sync(0xffffffffu, on);
        if (on) {
            const int q = __popc(m & ((1u << t) - 1u));
            day[q] = t;
            u0s[q] = u0;
            rcp[q] = 1.0 / u0;
        }
        if (t == 0) nday = __popc(m);
        if (t < nc && !on) dnvflux[c0 + t] = dndiffv[c0 + t] + 0.0;
    }
    if (t < NSYS_V) {
        const int ng = t / D_NV, nw = t - ng * D_NV;
        sl[t] = sol[nw];
        wa[t] = ng < D_NG - 1 ? K.gweight[ng] : K.fzerov[nw];
        wb[t] = ng < D_NG - 1 ? 1.0 - K.fzerov[nw] : 1.0;
        at[t] = nw * D_NG + ng;
    }
    __syncthreads();
    const int n = nday * NSYS_V;
    for (int i0 = t; i0 < n; i0 += DSOL_MLP * DSOL_THREADS) {
        double dv[DSOL_MLP];
#pragma unroll
        for (int q = 0; q < DSOL_MLP; ++q) {
            const int i = i0 + q * DSOL_THREADS, c = i / NSYS_V;
            dv[q] = i < n ? detau[(size_t)(c0 + day[c]) * NSYS_V + (i - c * NSYS_V)] : 6.0;
        }
#pragma unroll
        for (int q = 0; q < DSOL_MLP; ++q) {
            const int i = i0 + q * DSOL_THREADS;
            if (i >= n) break;
            const int c = i / NSYS_V, e = i - c * NSYS_V;
            const double u0 = u0s[c], d = dv[q];
            double v = 0.0;
            if (d <= 5.0) {
                // the quotient and the exponential without their special cases
                // where the operands allow it (rt_fastmath.cuh)
                const bool usual = d > 0x1p-300 && u0 < 0x1p300;
                const double x = usual ? -quot(d, u0, rcp[c]) : -d / u0;
                const double w = fabs(x) < 700.0 ? exp_r(x) : mgcm_rt_exp(x);
                v = u0 * sl[e] * w * wa[e] * wb[e];
            }
            term[c * DSOL_ROW + at[e]] = v;
        }
    }
    __syncthreads();
    if (t < nday) {
        double ds = 0.0;
        for (int q = 0; q < NSYS_V; ++q) ds = ds + term[t * DSOL_ROW + q];
        dnvflux[c0 + day[t]] = dndiffv[c0 + day[t]] + ds;
    }
}
size_t dsolflux_ctas(int ncol) { return (size_t)(ncol + DSOL_COLS - 1) / DSOL_COLS; }

// Integer bins as the pipeline uses them, for the bit-exact check of
// tpindex (code/tpindex.f90:72-134) and of the Planck index INT(T*10-499)
// (code/sfluxi.f90:54-55, code/gfluxi.f90:73-74,86-87).  Reads the column
// blocks rt_stage wrote -- each level's k-table corner offset and NH2O step
// -- and turns them back into MT, MP, NH2O; copies WRATIO and LCOEF(1..4);
// and evaluates planck_index, the function rt_stage uses, on every TLEV.
// One thread per (column, level K = 1..LEV); outputs [ncol][LEV] (LCOEF
// [ncol][LEV][4]); level 1 has no tpindex call and gets zeros.
__global__ void rt_bins_decode(const SegTable *__restrict__ st, int ncol, int max_nl,
                               const unsigned char *__restrict__ blocks, size_t stride,
                               uint32_t *status, int *__restrict__ mt, int *__restrict__ mp,
                               int *__restrict__ nh, int *__restrict__ npl, double *__restrict__ wr,
                               double *__restrict__ lk) {
    const SegDev &sg = st->seg[0];
    const int LEV = 2 * sg.L + 3;
    const long long n = (long long)ncol * LEV;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(i / LEV), k = (int)(i % LEV) + 1;
        npl[i] = planck_index(sg.tlev[(size_t)c * LEV + k - 1], status);
        if (k == 1) {
            mt[i] = mp[i] = nh[i] = 0;
            wr[i] = 0.0;
            for (int q = 0; q < 4; ++q) lk[i * 4 + q] = 0.0;
            continue;
        }
        const ColSmem s = carve_smem(const_cast<unsigned char *>(blocks) + (size_t)c * stride, max_nl,
                                     nullptr, false);
        const KLevel &r = s.klev[k];
        const int e = r.kofs / D_NGK;   // ((MT-1)*NP + MP-1)*NH + NH2O-1
        nh[i] = e % D_NH + 1;
        mp[i] = (e / D_NH) % D_NP + 1;
        mt[i] = e / (D_NH * D_NP) + 1;
        wr[i] = r.wr;
        for (int q = 0; q < 4; ++q) lk[i * 4 + q] = r.lk[q];
    }
}

}  // namespace mgcm

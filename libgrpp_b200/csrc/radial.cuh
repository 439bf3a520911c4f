// Radial integrals of the semilocal (type 2) and spin-orbit GRPP terms.
//
// Reference algorithm: libgrpp/radial_type2_integral.c:101-489 and
// libgrpp/screening.c:193-378. For one task (shells A, B, centre C) and each
// semilocal potential p of the centre, the table
//   Q_p[l1][l2][N] = int_0^inf U_p(r) F^A_l1(r) F^B_l2(r) r^N dr,
//   F_l(r) = sum_i c_i N_i exp(-a_i (r-CA)^2) M_l(2 a_i CA r),
// with l1 <= L_p + la, l2 <= L_p + lb, N <= la + lb, is computed by
//   * the one-centre analytic formula when CA = CB = 0;
//   * otherwise, per entry, the Shaw-Hill screening estimate (entries below
//     1e-16 return the estimate) and the nested Log3 quadrature
//     r_i = -5 ln(1 - x_i^3), levels of 31, 63, ..., 8191 points, stopping when
//     |S_L - S_{L-1}| <= 1e-16 unless |S|/|estimate| < 1e-3, capped at 8191 points.
//
// GPU mapping:
//  * radial_screen_unit_kernel: one warp per run of entries of one (task, potential), lanes over
//    entries, triples that cannot matter dropped first; the gate decisions are
//    libgrpp's. One-centre tasks get their analytic table (radial_one_centre_kernel).
//  * radial_walk_group_kernel: the grid walk of the tasks that have entries left, over tabulated
//    integrands, a thread per group of entries.
//  * radial_screen_kernel and radial_walk_kernel: the same by single entries and without tables
//    (no-allocation path; the walk also for batches whose tables would be too large). One CTA
//    per task; the grid is walked in chunks of one point per thread; a point's integrand values
//      w U_p(r) for every potential, F^A_l, F^B_l for every order, r^N,
//    are evaluated once and shared by all potentials and entries; every thread then advances
//    the running sums of the entries it owns, point by point in the reference's order and
//    association ((((w U) F1) F2) r^N).
#pragma once

#include "grpp_common.cuh"
#include "specfunc.cuh"
#include "exp_rn.h"

namespace grpp {

constexpr int kRadThreads = 128;
constexpr int kRadMaxPrims = 64;     // primitives per shell on the radial path
constexpr int kRadMaxPots = 24;      // semilocal potentials per centre
constexpr int kRadMaxTerms = 256;    // potential terms per centre (all semilocal potentials)
constexpr int kRadMaxLam = 24;       // lambda <= L + l
constexpr int kRadMaxN = 24;         // N <= la + lb
constexpr int kRadMaxLevel = 8;      // 8191 points
constexpr int kRadMaxEntries = 16384;

// entry flag bits
constexpr uint8_t kEntActive = 1, kEntScrOk = 2;

// A run of used entries of one semilocal potential of one task, screened by one warp of
// radial_screen_unit_kernel (or, for a one-centre task, evaluated by radial_one_centre_kernel):
// item, potential index, offset of the potential's (l1, l2, N) box within the item's table, offset of the run in ulist,
// number of entries.
struct ScrUnit {
    int item, pot, pe, uo, ne;
};

struct RadialArgs {
    int n_items;
    int64_t n_entries;          // total entries of all items (flat screening)
    const int *item_task;
    const int *task_a, *task_b, *task_c;
    const int *shell_L;
    const double *shell_origin;
    // shrunk (|c| > 1e-14) primitives with the normalisation folded in (radial_type2_integral.c:164-172)
    const int *rp_off, *rp_n;
    const double *rp_coef, *rp_alpha;
    // unshrunk primitives (one-centre branch, radial_type2_integral.c:126-155)
    const int *shell_nprim, *shell_prim_off;
    const double *prim_coef, *prim_alpha;
    const double *centre_origin;
    const int *centre_grpp;
    const int *grpp_sl_off, *grpp_sl_n, *sl_pot;
    const int *pot_L, *pot_nprim, *pot_prim_off, *pot_powers;
    const double *pot_coef, *pot_alpha;
    const int64_t *q_off;       // per item
    // walk: two lists of active entry indices (uint16) of up to list_max entries each, after
    // chunk_doubles doubles of point arrays in dynamic shared memory; list_max = 0: no lists
    int list_max, chunk_doubles;
    // w U_p(r) at every grid point per GRPP and semilocal potential slot, at
    // wu[(grpp * wu_npot + slot) * kRadGridPts + point] (wu_table_kernel); null: the walk
    // evaluates the potential terms itself
    const double *wu;
    int wu_npot;
    // F_l(r) = sum_i c_i N_i exp(-a_i (r-CS)^2) M_l(2 a_i CS r), l = 0..fp_lmax[k], at every grid
    // point for each (shell, centre) pair k of the batch (ftab_kernel), at
    // ftab[fp_off[k] + l * kRadGridPts + point]; item_fa / item_fb: the pairs (A, C) and (B, C)
    // of an item. ftab null: the walk evaluates F itself
    const double *ftab;
    const int64_t *fp_off;
    const int *fp_shell, *fp_centre, *fp_lmax, *item_fa, *item_fb;
    int n_fpairs;
    // entries the angular sums read: offsets within a potential's (l1, l2, N) block, per class
    // (L, la, lb) one list
    const uint16_t *ulist;
    // screening: runs of entries of one (task, potential) for radial_screen_unit_kernel, popped
    // from *scr_queue (zeroed before the launch); scr_lw: orders 0..scr_lw-1 of its Bessel tables
    const ScrUnit *scr_units;
    int n_scr_units, scr_lw;
    int *scr_queue;
    // runs of one-centre tasks, with prefix entry offsets su_off (radial_one_centre_kernel)
    const ScrUnit *su;
    const int64_t *su_off;
    int n_su;
    int64_t n_su_entries;
    double *Q;                  // table values (running sums during the walk)
    double *S_prev, *scr;       // per entry scratch, same indexing as Q
    uint8_t *eflag;             // per entry: kEntActive | kEntScrOk
    uint8_t *walk;              // per item: 1 if the grid walk has work
    int8_t *stop_level;         // per item: deepest level walked (learning labels), may be null
    const int8_t *pred_level;   // per item: predicted level (learned mode), may be null
    int *fallback_count;        // learned mode: items that needed more than predicted+1
    // learned mode: the walk pops items from this order (deepest predicted level first)
    const int *order;           // may be null: static round-robin over all items
    const int *n_order;
    int *queue;
    int *status;
    // operation counters (accumulated per CTA, one atomic add per item), see kRadCnt*
    unsigned long long *counters;
};

// counter slots: the FLOP model of the radial path is built from these counts
enum RadialCounter {
    kRadCntScreenCycles = 0,   // SM clock cycles spent in screening (sum over CTAs)
    kRadCntQuadCycles,         // SM clock cycles spent in the grid walk
    kRadCntItems,              // tasks through the grid walk
    kRadCntPoints,             // integrand points evaluated
    kRadCntBessel,             // M_l(x) evaluations of the integrand (points x prims x orders)
    kRadCntPrimPts,            // primitive Gaussians evaluated (points x prims)
    kRadCntTermPts,            // potential terms evaluated (points x terms)
    kRadCntPowPts,             // r^N evaluations (points x (la+lb+1))
    kRadCntAccum,              // entry x point accumulations
    kRadCntScrCombos,          // primitive screening estimates started
    kRadCntScrIters,           // fixed-point iterations of the screening
    kRadCntScrFinal,           // screening envelopes evaluated
    kRadCntLevels,             // grid levels walked (sum over tasks)
    kRadCntMmdTriples,         // type 1 / overlap primitive triples evaluated (mmd_kernel)
    kRadCntMmdFlops,           // their FP64 operations by the model of mmd_kernel's counting
    kRadCntNum
};

struct RadialShared {
    double CA, CB;
    int la, lb, np_a, np_b, npot, nterm_tot, d_n;
    int l1max_all, l2max_all;
    int one_centre;
    int grpp;
    int64_t fa_off, fb_off;  // F tables of (A, C) and (B, C), when tabulated
    int n_entries;
    int any_active;
    double ca[kRadMaxPrims], xa[kRadMaxPrims], ka[kRadMaxPrims];
    double cb[kRadMaxPrims], xb[kRadMaxPrims], kb[kRadMaxPrims];
    int pL[kRadMaxPots], pn[kRadMaxPots], poff[kRadMaxPots], pent[kRadMaxPots + 1];
    int tpow[kRadMaxTerms];
    double tcoef[kRadMaxTerms], talpha[kRadMaxTerms];
};

// ---- screening (screening.c:243-362) ------------------------------------------

// M_a(x) / M_b(x) for the adjacent orders (a, b) = (1, 0) if l = 0, else (l-1, l), both
// from one table row (screening.c:332-346 evaluates them as two separate calls)
__device__ __noinline__ double scr_ratio(int l, double x)
{
    const int na = l == 0 ? 1 : l - 1, nb = l == 0 ? 0 : l;
    if (x <= 1e-7) return bessel_small(na, x) / bessel_small(nb, x);
    if (x <= 16.0) {
        const int i0 = (int)(round(x * 100) + 1e-5);
        const double dx = x - i0 * 0.01;
        const double *row = c_tab.bessel + (size_t)i0 * kBesL * 5;
        return taylor4(row + 5 * na, dx) / taylor4(row + 5 * nb, dx);
    }
    return bessel_asym(na, x) / bessel_asym(nb, x);
}

__device__ __noinline__ double bessel_scaled_nl(int n, double x) { return bessel_scaled(n, x); }

// returns true on failure; *val is the primitive estimate
__device__ inline bool scr_prim(int l1, int l2, int n, double CA2, double CB2, double aA, double aB, double k1,
                                double k2, double eta, double *val, int *iters)
{
    *val = 0.0;
    *iters = 0;
    if (l1 >= 1 && fabs(k1) <= kZeroThresh) return false;
    if (l2 >= 1 && fabs(k2) <= kZeroThresh) return false;
    const double p = aA + aB + eta, CA = sqrt(CA2), CB = sqrt(CB2);
    if (l1 == 0 && l2 == 0 && fabs(k1) <= kZeroThresh && fabs(k2) <= kZeroThresh) {
        double gi;
        if (n % 2 == 0) {
            int k = n / 2;
            gi = dfact(2 * k - 1) / (pow(2.0, k + 1) * pow(p, k)) * sqrt(kPi / p);
        } else {
            int k = (n - 1) / 2;
            double f = 1.0;
            for (int q = 2; q <= k; q++) f *= q;
            gi = f / (2.0 * pow(p, k + 1));
        }
        *val = exp(-aA * CA * CA - aB * CB * CB) * gi;
        return false;
    }
    double r0 = (aA * CA + aB * CB) / p, r0p;
    int steps = 0;
    do {
        steps++;
        if (steps == 5) {
            *val = 0.0;
            return true;
        }
        r0p = r0;
        const double x1 = k1 * r0, x2 = k2 * r0;
        double a = scr_ratio(l1, x1) * x1 + scr_ratio(l2, x2) * x2 + n;
        if (l1 > 0) a = a - l1 - 1;
        if (l2 > 0) a = a - l2 - 1;
        r0 = sqrt(a / (2.0 * p));
        *iters = steps;
    } while (fabs(r0 - r0p) > 1e-2);
    *val = sqrt(kPi / p) * pow(r0, n) * bessel_scaled_nl(l1, k1 * r0) * bessel_scaled_nl(l2, k2 * r0) *
           exp(-eta * r0 * r0 - aA * (r0 - CA) * (r0 - CA) - aB * (r0 - CB) * (r0 - CB)) * 0.5 * (1 + erf(sqrt(p) * r0));
    *iters = -*iters - 1;  // negative: the envelope was evaluated
    return false;
}

// x^n for a small non-negative integer n by binary powering (libgrpp calls pow(r0, n);
// the estimate only feeds threshold tests, and the two agree to a few ulps)
__device__ __forceinline__ double ipow(double x, int n)
{
    double r = 1.0, b = x;
    while (n) {
        if (n & 1) r *= b;
        b *= b;
        n >>= 1;
    }
    return r;
}

// M_a(x) and M_b(x) with (a, b) = (1, 0) if l = 0, else (l-1, l) (screening.c:329-346), up to
// a common factor: the numerator and denominator of the ratio the fixed-point step uses.
// Above x = 16 both are the asymptotic series sum_k c_k (-1/x)^k / (2x); the 1/(2x) factor
// cancels in the ratio and is left out, so one reciprocal of x serves both.
__device__ __forceinline__ void scr_ratio_parts(int l, double x, double &num, double &den)
{
    const int na = l == 0 ? 1 : l - 1, nb = l == 0 ? 0 : l;
    if (x <= 1e-7) {
        num = bessel_small(na, x);
        den = bessel_small(nb, x);
    } else if (x <= 16.0) {
        const int i0 = (int)(round(x * 100) + 1e-5);
        const double dx = x - i0 * 0.01;
        const double *row = c_tab.bessel + (size_t)i0 * kBesL * 5;
        num = taylor4(row + 5 * na, dx);
        den = taylor4(row + 5 * nb, dx);
    } else {
        const double ninv = -1.0 / x;
        const double *ca = c_tab.rfun + na * kRfunL, *cb = c_tab.rfun + nb * kRfunL;
        double pw = 1.0, sa = 0.0, sb = 0.0;
        const int kmax = na > nb ? na : nb;
        for (int k = 0; k <= kmax; k++) {
            if (k <= na) sa += __ldg(ca + k) * pw;
            if (k <= nb) sb += __ldg(cb + k) * pw;
            pw *= ninv;
        }
        num = sa;
        den = sb;
    }
}

// Gaussian integral int_0^inf r^n exp(-p r^2) dr (screening.c:255-265): the
// screening estimate of two s functions on the centre and the one-centre analytic table
__device__ __forceinline__ double scr_gaussian_integral(int n, double p)
{
    if (n % 2 == 0) {
        const int k = n / 2;
        return dfact(2 * k - 1) / (pow(2.0, k + 1) * pow(p, k)) * sqrt(kPi / p);
    }
    const int k = (n - 1) / 2;
    double f = 1.0;
    for (int q = 2; q <= k; q++) f *= q;
    return f / (2.0 * pow(p, k + 1));
}

// T_l(x) = x M_(l-1)(x) / M_l(x), T_0(x) = x M_1(x) / M_0(x): what the fixed-point step of
// screening.c:329-362 takes of each side. Tabulated (tables.cpp) as Taylor coefficients in x up to
// x = 16 and of T_l - x in y = 1/x above, so a step costs one short polynomial per side and no
// division (two Taylor sums or asymptotic series per side and a division before); relative error
// below 3e-12 at every order. Below x = 1.25 libgrpp's own 4th-order
// Taylor sums of M_l lose digits (down to 0/0 for high l near 0, an undefined estimate): there
// its quotient is formed as libgrpp does. inv_x: 1/x, read for x > 16 only. An undefined
// estimate leaves r0 NaN (the entry is then walked): no table row is taken from a NaN, and scr_row
// keeps every row number inside its table.
__device__ __forceinline__ int scr_row(double g, unsigned n) { return (int)min(__double2uint_rz(g), n - 1u); }
__device__ __forceinline__ double scr_poly(const double *c, double h)
{
    return __ldg(c) + h * (__ldg(c + 1) + h * (__ldg(c + 2) + h * (__ldg(c + 3) + h * __ldg(c + 4))));
}
__device__ __forceinline__ double scr_t(int l, double x, double inv_x)
{
    if (!(x >= kRatXmin)) {
        double num, den;
        scr_ratio_parts(l, x, num, den);
        return num * x / den;
    }
    // one polynomial for both ranges, so that lanes on either side of 16 stay together
    const bool lo = x <= 16.0;
    const int i = scr_row(lo ? x * 100.0 + 0.5 : inv_x * kRatYInv + 0.5, lo ? kBesNX : kRatYN);
    const double h = lo ? x - i * 0.01 : inv_x - i * (1.0 / kRatYInv);
    return (lo ? 0.0 : x) + scr_poly((lo ? c_tab.ratio : c_tab.ratio_y) + (i * kRatL + l) * 5, h);
}
// M_l(x) of the envelope: Taylor in x up to 16, above of 2x M_l (a polynomial of degree l in 1/x) in y = 1/x
__device__ __forceinline__ double scr_m(int l, double x, double inv_x)
{
    const bool lo = x <= 16.0;
    const int i = scr_row(lo ? x * 100.0 + 0.5 : inv_x * kBesYInv + 0.5, lo ? kBesNX : kBesYN);
    const double h = lo ? x - i * 0.01 : inv_x - i * (1.0 / kBesYInv);
    return scr_poly((lo ? c_tab.bes_t : c_tab.bes_y) + (i * kRatL + l) * 5, h) * (lo ? 1.0 : 0.5 * inv_x);
}

// The envelope of screening.c:308-318 at the fixed point r0, with sqpi = sqrt(pi / p) and
// sqp = sqrt(p). Every factor is finite and non-negative where the Gaussian factor is positive; one that
// underflowed to exactly 0 makes the product exactly 0, and a NaN one (r0 undefined) makes it NaN, so the other
// factors are not needed there; and 1 + erf(z) is
// exactly 2 once erfc(z) < 2^-54 (z > 5.9), taken here as p r0^2 > 36 (z > 6). The product keeps
// libgrpp's order (screening.c:333-338).
__device__ __forceinline__ double scr_envelope(int l1, int l2, int n, double CA, double CB, double aA, double aB,
                                               double eta, double p, double k1, double k2, double ik1, double ik2,
                                               double r0, double sqpi, double sqp)
{
    const double e1 = r0 - CA, e2 = r0 - CB;
    const double ex = exp(-eta * r0 * r0 - aA * e1 * e1 - aB * e2 * e2);
    if (!(ex > 0.0)) return ex;
    const double z2 = p * r0 * r0;
    const double erf_part = z2 > 36.0 ? 2.0 : 1 + erf(sqp * r0);
    const double ir = 1.0 / r0;
    return sqpi * ipow(r0, n) * scr_m(l1, k1 * r0, ik1 * ir) * scr_m(l2, k2 * r0, ik2 * ir) * ex * 0.5 * erf_part;
}

// The fixed-point update of screening.c:329-362: r0'^2 = s / (2p),
// s = T_l1(x1) + T_l2(x2) + n - (l1 + 1 if l1 > 0) - (l2 + 1 if l2 > 0); cn = n - (..) - (..)
__device__ __forceinline__ double scr_next(double t1, double t2, int cn, double inv2p) { return (t1 + t2 + cn) * inv2p; }

// One-centre entry (CA = CB = 0): libgrpp's analytic table (radial_type2_integral.c:126-155),
// only l1 = l2 = 0 non-zero
__device__ double scr_one_centre_entry(const RadialArgs &a, int sa, int sb, int la, int lb, int l1, int l2, int N,
                                       int nk, int po)
{
    if (l1 != 0 || l2 != 0) return 0.0;
    const int na = __ldg(a.shell_nprim + sa), nb = __ldg(a.shell_nprim + sb);
    const double *pca = a.prim_coef + __ldg(a.shell_prim_off + sa), *pxa = a.prim_alpha + __ldg(a.shell_prim_off + sa);
    const double *pcb = a.prim_coef + __ldg(a.shell_prim_off + sb), *pxb = a.prim_alpha + __ldg(a.shell_prim_off + sb);
    double v = 0.0;
    for (int i = 0; i < na; i++) {
        const double ci = __ldg(pca + i) * gaussian_norm(la, __ldg(pxa + i));
        for (int j = 0; j < nb; j++) {
            const double cj = __ldg(pcb + j) * gaussian_norm(lb, __ldg(pxb + j));
            for (int k = 0; k < nk; k++) {
                const double pp = __ldg(pxa + i) + __ldg(pxb + j) + __ldg(a.pot_alpha + po + k);
                const double f = ci * cj * __ldg(a.pot_coef + po + k);
                v += f * scr_gaussian_integral(__ldg(a.pot_powers + po + k) + N, pp);
            }
        }
    }
    return v;
}

// libgrpp's decision for a screened entry (radial_type2_integral.c:264-279): an estimate below
// 1e-16 is the entry's value; otherwise the entry is walked, with forced refinement only when
// the estimate is valid
__device__ __forceinline__ void scr_store(const RadialArgs &a, int item, int64_t g, double sum, bool fail)
{
    a.scr[g] = sum;
    if (!fail && fabs(sum) < 1e-16) {
        a.Q[g] = sum;
        a.eflag[g] = kEntScrOk;
    } else {
        a.Q[g] = 0.0;
        a.eflag[g] = kEntActive | (fail ? 0 : kEntScrOk);
        a.walk[item] = 1;
    }
}

// Whether a triple's estimate is below 1e-40 and its iteration ends at the first step, for every
// entry with l1 <= l1m, l2 <= l2m and N between nlo and nhi (pw: the term's power; c: the triple's
// coefficient). The bounds on the Bessel ratios hold for the tabulated values too when their
// arguments are at least 0.5 (or the side's distance is 0, where entries with l > 0 are 0) and
// the orders at most 16: their relative error is then below 1e-6, against a margin of 0.5%.
__device__ __forceinline__ bool scr_dead(double CA, double CB, double aA, double aB, double eta, double c, int pw, int l1m,
                                         int l2m, int nlo, int nhi)
{
    const double p = aA + aB + eta, inv_p = 1.0 / p, inv2p = 0.5 * inv_p;
    const double r = (aA * CA + aB * CB) * inv_p, k1 = 2 * aA * CA, k2 = 2 * aB * CB;
    const bool in1 = k1 * r >= 0.5, in2 = k2 * r >= 0.5;
    if (!(in1 || k1 <= kZeroThresh) || !(in2 || k2 <= kZeroThresh) || !(in1 || in2) || l1m > 16 || l2m > 16) return false;
    if (!((nhi + pw + l1m + l2m) * inv2p <= 0.0199 * r + 0.99e-4) || !((2 - nlo - pw) * inv2p <= 0.0199 * r - 1e-4)) return false;
    const double eA = r - CA, eB = r - CB;
    const float g = (float)(-eta * r * r - aA * eA * eA - aB * eB * eB);
    const float cm = (float)fabs(c);  // NaN stays NaN: such a triple is kept, as an infinite one is
    const float b = 0.5f * __logf(3.1416f * (float)inv_p) + (nhi + pw) * __logf(fmaxf(1.f, (float)r + 0.01f)) +
                    __logf(cm <= 1e-37f ? 1e-37f : cm);
    return g + b < -92.f;
}

#ifndef GRPP_RADIAL_TABLES_ONLY
// Entries of one-centre tasks (CA = CB = 0): libgrpp's analytic table, one thread per entry over
// the flattened runs of a.su.
__global__ void __launch_bounds__(kRadThreads) radial_one_centre_kernel(RadialArgs a)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t gu = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; gu < a.n_su_entries; gu += stride) {
        int lo = 0, hi = a.n_su - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(a.su_off + mid) <= gu) lo = mid;
            else hi = mid - 1;
        }
        const ScrUnit &U = a.su[lo];
        const int e = a.ulist[U.uo + (int)(gu - __ldg(a.su_off + lo))];
        const int t = __ldg(a.item_task + U.item), sa = __ldg(a.task_a + t), sb = __ldg(a.task_b + t);
        const int la = __ldg(a.shell_L + sa), lb = __ldg(a.shell_L + sb), dn = la + lb + 1;
        const int d2 = __ldg(a.pot_L + U.pot) + lb + 1, l1 = e / (d2 * dn), rem = e - l1 * d2 * dn, l2 = rem / dn;
        const int64_t g = __ldg(a.q_off + U.item) + U.pe + e;
        a.Q[g] = scr_one_centre_entry(a, sa, sb, la, lb, l1, l2, rem - l2 * dn, __ldg(a.pot_nprim + U.pot),
                                      __ldg(a.pot_prim_off + U.pot));
        a.eflag[g] = 0;
    }
}

// ---- screening: radial_screen_unit_kernel ------------------------------------------------------
//
// A warp screens one run of entries (l1, l2, N) of one (task, semilocal potential): for each entry
// libgrpp's estimate, the sum over primitive triples (i, j, k) of c times a primitive estimate
// (screening.c:193-220, 243-362), which decides whether the entry is walked.
//
//  * Triples that cannot matter are dropped first, for the whole run. The primitive estimate is
//    an envelope at the fixed point r' of r'^2 = r^2 + c / (2p), started at r = (a_A CA + a_B CB)/p;
//    the Bessel ratios obey x - 1 <= x M_(l-1)/M_l - l - 1 <= x + l, so n - 2 <= c <= n + l1 + l2.
//    When both ends keep |r' - r| below 1e-2, libgrpp's iteration stops after one step and cannot
//    fail; and the envelope is at most sqrt(pi/p) max(1, r + 0.01)^n times the Gaussian factor at
//    r, its largest value. Where that bound times |c| is below e^-92 = 1e-40 the triple cannot
//    change a sum that is compared with 1e-16 (scr_dead). This removes two thirds of the triples
//    of the 64-atom s..g workload and half of those of a 15-atom molecule.
//  * The remaining triples are staged in shared memory, 32 at a time: everything that does not
//    depend on the entry, including the first step's T_l of every order (its arguments k r do
//    not depend on the entry).
//  * Lanes take entries, each walking the staged triples in order; where the run's entries leave
//    lanes idle each entry gets a group of G = 2, 4 or 8 lanes that share its triples (values added by a
//    shuffle tree; the sum's order then differs from libgrpp's in the last bits, which matter
//    only to an estimate within them of a threshold). More lanes per entry would spread the
//    Bessel table reads over as many rows. A triple that fails ends the entry (it is then walked).
// What bounds it: FP64 latency with about half of the lanes active (entries need different
// numbers of steps). Five blocks per SM (96 registers) against four and six: 17.4, 18.3, 16.9 ms
// on the 65536 tasks of the s..g workload, where the previous pair of kernels (a thread per entry,
// every triple, two Bessel sums per side and a division per step) took 49.5 ms; the matrices
// of a 15-atom molecule 24.7 -> 12.8 ms, of three atoms 1.24 -> 0.44 ms. Lanes over triples
// throughout (32 per entry) measured 53.7 ms on the first: the table rows of 32 different
// arguments do not stay in L1.
constexpr int kScrWarps = 4;    // warps per block, each on its own run
constexpr int kScrRunMax = 64;  // entries per run
constexpr int kScrArr = 13;     // staged scalars per triple
// shared memory of a warp, in doubles: T_l [side][order][32], scalars, sums, then ints
// (r power, waiting triples, failed entries)
__host__ __device__ inline int scr_warp_doubles(int lw) { return 2 * lw * 32 + kScrArr * 32 + kScrRunMax + (32 + 64 + kScrRunMax) / 2; }

__global__ void __launch_bounds__(32 * kScrWarps, 5) radial_screen_unit_kernel(RadialArgs a)
{
    extern __shared__ double scr_sm[];
    const int lane = threadIdx.x & 31, lw = a.scr_lw;
    double *PA = scr_sm + (threadIdx.x >> 5) * scr_warp_doubles(lw), *PB = PA + lw * 32;
    double *t_aA = PB + lw * 32, *t_aB = t_aA + 32, *t_eta = t_aB + 32, *t_p = t_eta + 32, *t_i2p = t_p + 32, *t_sqpi = t_i2p + 32,
           *t_sqp = t_sqpi + 32, *t_k1 = t_sqp + 32, *t_k2 = t_k1 + 32, *t_r0 = t_k2 + 32, *t_ik1 = t_r0 + 32, *t_ik2 = t_ik1 + 32,
           *t_c = t_ik2 + 32, *s_sum = t_c + 32;
    int *t_pw = (int *)(s_sum + kScrRunMax), *list = t_pw + 32, *s_bad = list + 64;
    const long long t0 = clock64();
    unsigned long long c_combo = 0, c_iter = 0, c_final = 0;
    for (;;) {
        int u = 0;
        if (lane == 0) u = atomicAdd(a.scr_queue, 1);
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= a.n_scr_units) break;
        const ScrUnit U = a.scr_units[u];
        const int item = U.item, pot = U.pot, ne = U.ne;
        const int t = __ldg(a.item_task + item);
        const int sa = __ldg(a.task_a + t), sb = __ldg(a.task_b + t), c = __ldg(a.task_c + t);
        const double *Ao = a.shell_origin + 3 * sa, *Bo = a.shell_origin + 3 * sb, *Co = a.centre_origin + 3 * c;
        double CA2 = 0.0, CB2 = 0.0;
        for (int d = 0; d < 3; d++) {
            const double uu = __ldg(Co + d) - __ldg(Ao + d), vv = __ldg(Co + d) - __ldg(Bo + d);
            CA2 += uu * uu;
            CB2 += vv * vv;
        }
        const double CA = sqrt(CA2), CB = sqrt(CB2);
        const int la = __ldg(a.shell_L + sa), lb = __ldg(a.shell_L + sb), dn = la + lb + 1;
        const int Lp = __ldg(a.pot_L + pot), d2 = Lp + lb + 1;
        const int nk = __ldg(a.pot_nprim + pot), po = __ldg(a.pot_prim_off + pot);
        const int na = __ldg(a.rp_n + sa), nb = __ldg(a.rp_n + sb), T = na * nb * nk;
        const double *ca = a.rp_coef + __ldg(a.rp_off + sa), *xa = a.rp_alpha + __ldg(a.rp_off + sa);
        const double *cb = a.rp_coef + __ldg(a.rp_off + sb), *xb = a.rp_alpha + __ldg(a.rp_off + sb);
        const int64_t g0 = __ldg(a.q_off + item) + U.pe;
        __syncwarp();  // the previous run's shared arrays are consumed
        int l1m = 0, l2m = 0, nlo = dn, nhi = 0;
        for (int q = lane; q < ne; q += 32) {
            const int e = a.ulist[U.uo + q], l1 = e / (d2 * dn), rem = e - l1 * d2 * dn, l2 = rem / dn, N = rem - l2 * dn;
            l1m = max(l1m, l1);
            l2m = max(l2m, l2);
            nlo = min(nlo, N);
            nhi = max(nhi, N);
            s_sum[q] = 0.0;
            s_bad[q] = 0;
        }
        l1m = __reduce_max_sync(0xffffffffu, l1m);
        l2m = __reduce_max_sync(0xffffffffu, l2m);
        nlo = __reduce_min_sync(0xffffffffu, nlo);
        nhi = __reduce_max_sync(0xffffffffu, nhi);
        // lanes per entry: the fewest that leave at most an eighth of the lanes without an entry
        int lg = 0;
        while (lg < 3 && ((ne + (32 >> lg) - 1) & ~((32 >> lg) - 1)) * 7 > 8 * ne) lg++;
        const int G = 1 << lg;
        int pos = 0, nl = 0;
        unsigned n_dead = 0;
        for (;;) {
            // the next triples in libgrpp's (i, j, k) order that are not dropped
            while (nl < 32 && pos < T) {
                const int q = pos + lane;
                bool live = false;
                if (q < T) {
                    const int i = q / (nb * nk), r = q - i * nb * nk, j = r / nk, k = r - j * nk;
                    live = !scr_dead(CA, CB, __ldg(xa + i), __ldg(xb + j), __ldg(a.pot_alpha + po + k),
                                     __ldg(ca + i) * __ldg(cb + j) * __ldg(a.pot_coef + po + k), __ldg(a.pot_powers + po + k), l1m,
                                     l2m, nlo, nhi);
                }
                const unsigned m = __ballot_sync(0xffffffffu, live);
                if (live) list[nl + __popc(m & ((1u << lane) - 1))] = q;
                n_dead += min(32, T - pos) - __popc(m);
                nl += __popc(m);
                pos += 32;
            }
            if (nl == 0) break;
            const int nc = min(32, nl);
            __syncwarp();
            if (lane < nc) {
                const int q = list[lane], i = q / (nb * nk), r = q - i * nb * nk, j = r / nk, k = r - j * nk;
                const double aA = __ldg(xa + i), aB = __ldg(xb + j), eta = __ldg(a.pot_alpha + po + k);
                const double k1 = 2 * aA * CA, k2 = 2 * aB * CB;
                const double p = aA + aB + eta, inv_p = 1.0 / p;
                const double r0 = (aA * CA + aB * CB) * inv_p;
                t_aA[lane] = aA;
                t_aB[lane] = aB;
                t_eta[lane] = eta;
                t_p[lane] = p;
                t_i2p[lane] = 0.5 * inv_p;
                t_sqpi[lane] = sqrt(kPi * inv_p);
                t_sqp[lane] = sqrt(p);
                t_k1[lane] = k1;
                t_k2[lane] = k2;
                t_r0[lane] = r0;
                t_ik1[lane] = 1.0 / k1;
                t_ik2[lane] = 1.0 / k2;
                t_c[lane] = __ldg(ca + i) * __ldg(cb + j) * __ldg(a.pot_coef + po + k);
                t_pw[lane] = __ldg(a.pot_powers + po + k);
                const double i1 = 1.0 / (k1 * r0), i2 = 1.0 / (k2 * r0);
                for (int l = 0; l <= l1m; l++) PA[l * 32 + lane] = scr_t(l, k1 * r0, i1);
                for (int l = 0; l <= l2m; l++) PB[l * 32 + lane] = scr_t(l, k2 * r0, i2);
            }
            __syncwarp();
            for (int e0 = 0; e0 < ne; e0 += 32 >> lg) {
                const int ei = e0 + (lane >> lg);
                const bool on = ei < ne && !s_bad[ei < ne ? ei : 0];
                const int e = a.ulist[U.uo + (ei < ne ? ei : 0)];
                const int l1 = e / (d2 * dn), rem = e - l1 * d2 * dn, l2 = rem / dn, N = rem - l2 * dn;
                const int cl = N - (l1 > 0 ? l1 + 1 : 0) - (l2 > 0 ? l2 + 1 : 0);
                double sum = 0.0;
                bool fail = false;
                for (int q0 = 0; q0 < nc; q0 += G) {
                    const int q = q0 + (lane & (G - 1));
                    const bool go = on && !fail && q < nc;
                    const double k1 = t_k1[q & 31], k2 = t_k2[q & 31], p = t_p[q & 31];
                    const bool z1 = fabs(k1) <= kZeroThresh, z2 = fabs(k2) <= kZeroThresh, ss = l1 == 0 && l2 == 0 && z1 && z2;
                    bool step = go && !(l1 >= 1 && z1) && !(l2 >= 1 && z2) && !ss, conv = false;
                    const int pw = t_pw[q & 31], n = N + pw;
                    c_combo += go;
                    double r0 = 0.0;
                    if (step) {
                        const double inv2p = t_i2p[q], ik1 = t_ik1[q], ik2 = t_ik2[q];
                        double r0p = t_r0[q];
                        r0 = sqrt(scr_next(PA[l1 * 32 + q], PB[l2 * 32 + q], cl + pw, inv2p));
                        int steps = 1;
                        while (fabs(r0 - r0p) > 1e-2 && steps < 4) {
                            steps++;
                            r0p = r0;
                            const double ir = 1.0 / r0;  // a factor of both sides' 1/x
                            r0 = sqrt(scr_next(scr_t(l1, k1 * r0, ik1 * ir), scr_t(l2, k2 * r0, ik2 * ir), cl + pw, inv2p));
                        }
                        c_iter += steps;
                        fail = fabs(r0 - r0p) > 1e-2;  // no fixed point in four steps
                        conv = !fail;
                    }
                    __syncwarp();
                    if (conv) {
                        c_final++;
                        sum += t_c[q] * scr_envelope(l1, l2, n, CA, CB, t_aA[q], t_aB[q], t_eta[q], p, k1, k2, t_ik1[q], t_ik2[q], r0,
                                                     t_sqpi[q], t_sqp[q]);
                    } else if (go && ss) {
                        sum += t_c[q] * exp(-t_aA[q] * CA * CA - t_aB[q] * CB * CB) * scr_gaussian_integral(n, p);
                    }
                    __syncwarp();
                }
                const unsigned bad = __ballot_sync(0xffffffffu, fail) >> (lane & ~(G - 1)) & ((1u << G) - 1);
                for (int o = G >> 1; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                if (on && (lane & (G - 1)) == 0) {
                    s_sum[ei] += sum;
                    if (bad) s_bad[ei] = 1;
                }
                __syncwarp();
            }
            // the triples that still wait move to the front
            const int rest = nl - nc;
            const int keep = lane < rest ? list[nc + lane] : 0;
            __syncwarp();
            if (lane < rest) list[lane] = keep;
            nl = rest;
            __syncwarp();
        }
        for (int q = lane; q < ne; q += 32) {
            scr_store(a, item, g0 + a.ulist[U.uo + q], s_sum[q], s_bad[q] != 0);
            if (!s_bad[q]) {  // a dropped triple is one step and one envelope of libgrpp's
                c_combo += n_dead;
                c_iter += n_dead;
                c_final += n_dead;
            }
        }
    }
    if (a.counters) {
        unsigned long long v[3] = {c_combo, c_iter, c_final};
        for (int k = 0; k < 3; k++)
            for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
        if (lane == 0) {
            atomicAdd(a.counters + kRadCntScrCombos, v[0]);
            atomicAdd(a.counters + kRadCntScrIters, v[1]);
            atomicAdd(a.counters + kRadCntScrFinal, v[2]);
            atomicAdd(a.counters + kRadCntScreenCycles, (unsigned long long)(clock64() - t0));
        }
    }
}

#endif  // GRPP_RADIAL_TABLES_ONLY

// decode entry index within an item -> (potential, l1, l2, N)
__device__ __forceinline__ void decode_entry(const RadialShared &sh, int e, int &p, int &l1, int &l2, int &N)
{
    p = 0;
    while (e >= sh.pent[p + 1]) p++;
    int r = e - sh.pent[p];
    const int d2 = sh.pL[p] + sh.lb + 1, dn = sh.d_n;
    l1 = r / (d2 * dn);
    r -= l1 * d2 * dn;
    l2 = r / dn;
    N = r - l2 * dn;
}

// Log3 point i of a grid of nr points (radial_type2_integral.c:357-365)
__device__ __forceinline__ void log3_point(int i, int nr, double &r, double &w)
{
    const double R = 5.0, R3 = R * R * R;
    const double xi = i / (nr + 1.0), xi3 = xi * xi * xi, ln = log(1 - xi3);
    w = 3 * R3 * xi * xi * ln * ln / ((1 - xi3) * (nr + 1.0));
    r = -R * ln;
}

// r and w of walk-order point f (point i of the level's nr-point grid): libgrpp's values from
// the host-built grid table (grpp_common.cuh) when present, else computed here
__device__ __forceinline__ void grid_point(int f, int i, int nr, double &r, double &w)
{
    if (c_tab.grid) {
        r = __ldg(c_tab.grid + (size_t)kGridRowR * kGridPts + f);
        w = __ldg(c_tab.grid + (size_t)kGridRowW * kGridPts + f);
    } else {
        log3_point(i, nr, r, w);
    }
}

// r^(n-2) of a potential term (n = 0, 1, 2) at walk-order point f: pow(r, n-2) from the grid
// table when present (potential.c:70-81), else 1/r^2, 1/r from the given reciprocals
__device__ __forceinline__ double grid_rpow_m2(int f, int pw, double ir, double ir2)
{
    if (pw == 2) return 1.0;
    if (c_tab.grid) return __ldg(c_tab.grid + (size_t)(pw == 1 ? kGridRowRinv : kGridRowRinv2) * kGridPts + f);
    return pw == 1 ? ir : ir2;
}


// task geometry, primitives and potential terms into shared memory
__device__ void load_task(const RadialArgs &a, int item, RadialShared &sh, int tid, int nthr)
{
    const int t = a.item_task[item];
    const int sa = a.task_a[t], sb = a.task_b[t], c = a.task_c[t];
    if (tid == 0) {
        const double *Ao = a.shell_origin + 3 * sa, *Bo = a.shell_origin + 3 * sb, *Co = a.centre_origin + 3 * c;
        double CAv[3], CBv[3];
        for (int d = 0; d < 3; d++) {
            CAv[d] = Co[d] - Ao[d];
            CBv[d] = Co[d] - Bo[d];
        }
        const double CA2 = CAv[0] * CAv[0] + CAv[1] * CAv[1] + CAv[2] * CAv[2];
        const double CB2 = CBv[0] * CBv[0] + CBv[1] * CBv[1] + CBv[2] * CBv[2];
        sh.one_centre = CA2 < 1e-14 && CB2 < 1e-14;
        sh.CA = sqrt(CA2);
        sh.CB = sqrt(CB2);
        sh.la = a.shell_L[sa];
        sh.lb = a.shell_L[sb];
        sh.d_n = sh.la + sh.lb + 1;
        const int g = a.centre_grpp[c];
        sh.grpp = g;
        sh.npot = a.grpp_sl_n[g];
        int e = 0, nt = 0, l1m = 0, l2m = 0;
        for (int p = 0; p < sh.npot; p++) {
            const int pot = a.sl_pot[a.grpp_sl_off[g] + p];
            sh.pL[p] = a.pot_L[pot];
            sh.pn[p] = a.pot_nprim[pot];
            sh.poff[p] = nt;
            for (int k = 0; k < sh.pn[p]; k++) {
                const int o = a.pot_prim_off[pot] + k;
                sh.tpow[nt] = a.pot_powers[o];
                sh.tcoef[nt] = a.pot_coef[o];
                sh.talpha[nt] = a.pot_alpha[o];
                nt++;
            }
            sh.pent[p] = e;
            e += (sh.pL[p] + sh.la + 1) * (sh.pL[p] + sh.lb + 1) * sh.d_n;
            l1m = max(l1m, sh.pL[p] + sh.la);
            l2m = max(l2m, sh.pL[p] + sh.lb);
        }
        sh.pent[sh.npot] = e;
        sh.n_entries = e;
        sh.nterm_tot = nt;
        sh.l1max_all = l1m;
        sh.l2max_all = l2m;
        sh.np_a = a.rp_n[sa];
        sh.np_b = a.rp_n[sb];
        if (a.ftab) {
            sh.fa_off = a.fp_off[a.item_fa[item]];
            sh.fb_off = a.fp_off[a.item_fb[item]];
        }
    }
    __syncthreads();
    for (int i = tid; i < sh.np_a; i += nthr) {
        sh.ca[i] = a.rp_coef[a.rp_off[sa] + i];
        sh.xa[i] = a.rp_alpha[a.rp_off[sa] + i];
        sh.ka[i] = 2.0 * sh.xa[i] * sh.CA;
    }
    for (int i = tid; i < sh.np_b; i += nthr) {
        sh.cb[i] = a.rp_coef[a.rp_off[sb] + i];
        sh.xb[i] = a.rp_alpha[a.rp_off[sb] + i];
        sh.kb[i] = 2.0 * sh.xb[i] * sh.CB;
    }
    __syncthreads();
}

// analytic one-centre entry (radial_type2_integral.c:126-155): only l1 = l2 = 0 is non-zero
__device__ double one_centre_entry(const RadialArgs &a, const RadialShared &sh, int sa, int sb, int p, int l1, int l2, int N)
{
    double v = 0.0;
    if (l1 != 0 || l2 != 0) return 0.0;
    const int na = a.shell_nprim[sa], nb = a.shell_nprim[sb];
    const double *pca = a.prim_coef + a.shell_prim_off[sa], *pxa = a.prim_alpha + a.shell_prim_off[sa];
    const double *pcb = a.prim_coef + a.shell_prim_off[sb], *pxb = a.prim_alpha + a.shell_prim_off[sb];
    for (int i = 0; i < na; i++) {
        const double ci = pca[i] * gaussian_norm(sh.la, pxa[i]);
        for (int j = 0; j < nb; j++) {
            const double cj = pcb[j] * gaussian_norm(sh.lb, pxb[j]);
            for (int k = 0; k < sh.pn[p]; k++) {
                const int tk = sh.poff[p] + k;
                const double pp = pxa[i] + pxb[j] + sh.talpha[tk];
                const double f = ci * cj * sh.tcoef[tk];
                const int n = sh.tpow[tk] + N;
                double gi;
                if (n % 2 == 0) {
                    const int kk = n / 2;
                    gi = dfact(2 * kk - 1) / (pow(2.0, kk + 1) * pow(pp, kk)) * sqrt(kPi / pp);
                } else {
                    const int kk = (n - 1) / 2;
                    double fct = 1.0;
                    for (int q = 2; q <= kk; q++) fct *= q;
                    gi = fct / (2.0 * pow(pp, kk + 1));
                }
                v += f * gi;
            }
        }
    }
    return v;
}

#ifndef GRPP_RADIAL_TABLES_ONLY
__global__ void __launch_bounds__(kRadThreads) radial_screen_kernel(RadialArgs a)
{
    __shared__ RadialShared sh;
    const int tid = threadIdx.x, lane = tid & 31;
    for (int item = blockIdx.x; item < a.n_items; item += gridDim.x) {
        __syncthreads();
        load_task(a, item, sh, tid, kRadThreads);
        const int t = a.item_task[item];
        const int sa = a.task_a[t], sb = a.task_b[t];
        const int64_t qo = a.q_off[item];
        double *Q = a.Q + qo, *SC = a.scr + qo;
        uint8_t *EF = a.eflag + qo;
        const int nE = sh.n_entries, np_a = sh.np_a, np_b = sh.np_b;
        const long long t0 = clock64();
        unsigned long long c_combo = 0, c_iter = 0, c_final = 0;
        int active = 0;
        if (sh.one_centre) {
            for (int e = tid; e < nE; e += kRadThreads) {
                int p, l1, l2, N;
                decode_entry(sh, e, p, l1, l2, N);
                Q[e] = one_centre_entry(a, sh, sa, sb, p, l1, l2, N);
                EF[e] = 0;
            }
        } else {
            const double CA2 = sh.CA * sh.CA, CB2 = sh.CB * sh.CB;
            for (int e = tid; e < nE; e += kRadThreads) {
                int p, l1, l2, N;
                decode_entry(sh, e, p, l1, l2, N);
                // screening.c:193-220: triples in (bra, ket, potential term) order, stop at the first failure
                double sum = 0.0;
                bool fail = false;
                const int nk = sh.pn[p];
                for (int i = 0; i < np_a && !fail; i++)
                    for (int j = 0; j < np_b && !fail; j++)
                        for (int k = 0; k < nk; k++) {
                            const int tk = sh.poff[p] + k;
                            double v;
                            int it;
                            const bool f = scr_prim(l1, l2, N + sh.tpow[tk], CA2, CB2, sh.xa[i], sh.xb[j], sh.ka[i],
                                                    sh.kb[j], sh.talpha[tk], &v, &it);
                            c_combo++;
                            if (it < 0) {
                                c_final++;
                                it = -it - 1;
                            }
                            c_iter += it;
                            if (f) {
                                fail = true;
                                break;
                            }
                            sum += sh.ca[i] * sh.cb[j] * sh.tcoef[tk] * v;
                        }
                SC[e] = sum;
                if (!fail && fabs(sum) < 1e-16) {
                    Q[e] = sum;
                    EF[e] = kEntScrOk;
                } else {
                    Q[e] = 0.0;
                    EF[e] = kEntActive | (fail ? 0 : kEntScrOk);
                    active = 1;
                }
            }
        }
        const int any = __syncthreads_or(active);
        if (tid == 0) {
            a.walk[item] = (uint8_t)any;
            if (a.stop_level) a.stop_level[item] = 0;
        }
        if (a.counters) {
            unsigned long long v[3] = {c_combo, c_iter, c_final};
            for (int k = 0; k < 3; k++)
                for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
            if (lane == 0) {
                atomicAdd(a.counters + kRadCntScrCombos, v[0]);
                atomicAdd(a.counters + kRadCntScrIters, v[1]);
                atomicAdd(a.counters + kRadCntScrFinal, v[2]);
            }
            if (tid == 0) atomicAdd(a.counters + kRadCntScreenCycles, (unsigned long long)(clock64() - t0));
        }
    }
}
#endif  // GRPP_RADIAL_TABLES_ONLY

// dst[l * stride] += e * M_l(x) for l = 0..lmax, one table row (specfunc_scaled_mod_sph_bessel.c:72-122)
__device__ __forceinline__ void bessel_row_acc(int lmax, double x, double e, double *dst, int stride)
{
    if (x <= 1e-7) {
#pragma unroll 1
        for (int l = 0; l <= lmax; l++) dst[l * stride] += e * bessel_small(l, x);
    } else if (x <= 16.0) {
        const int i0 = (int)(round(x * 100) + 1e-5);
        const double dx = x - i0 * 0.01;
        const double dx2 = dx * dx, dx3 = dx2 * dx, dx4 = dx3 * dx;
        // orders l, l+1 from one 80-byte block of the pair layout: five 16-byte loads
        const double2 *d = reinterpret_cast<const double2 *>(c_tab.bessel_p) + (size_t)i0 * kBesL * 5 / 2;
#pragma unroll 1
        for (int l = 0; l <= lmax; l += 2) {
            const double2 *q = d + 5 * (l / 2);
            const double2 c0 = __ldg(q), c1 = __ldg(q + 1), c2 = __ldg(q + 2), c3 = __ldg(q + 3), c4 = __ldg(q + 4);
            const double m0 = c0.x + c1.x * dx + c2.x * dx2 * 0.5 + c3.x * dx3 * (1.0 / 6.0) + c4.x * dx4 * (1.0 / 24.0);
            dst[l * stride] += e * m0;
            if (l < lmax) {
                const double m1 = c0.y + c1.y * dx + c2.y * dx2 * 0.5 + c3.y * dx3 * (1.0 / 6.0) + c4.y * dx4 * (1.0 / 24.0);
                dst[(l + 1) * stride] += e * m1;
            }
        }
    } else {
#pragma unroll 1
        for (int l = 0; l <= lmax; l++) dst[l * stride] += e * bessel_asym(l, x);
    }
}

constexpr int kRadRow = kRadThreads + 1;  // padded row stride of the chunk arrays (no bank conflicts)
constexpr int kRadGridPts = kGridPts;     // points of levels 0..8 together

// Level of point f of the nested grid in walk order (level 0: f = 0..30; level L >= 1:
// f = 2^(L+4)-1 .. 2^(L+5)-2), and the point's index i on that level's grid of nr points.
__device__ __forceinline__ void walk_point(int f, int &level, int &i, int &nr)
{
    const int lg = 31 - __clz(f + 1);  // floor(log2(f + 1))
    level = lg > 4 ? lg - 4 : 0;
    if (level == 0) {
        i = f + 1;
        nr = 31;
    } else {
        i = 2 * (f - ((1 << (level + 4)) - 1)) + 1;
        nr = (1 << (level + 5)) - 1;
    }
}

// last walk-order point of level L
__device__ __forceinline__ int level_last_point(int L) { return (1 << (L + 5)) - 2; }

// The nested Log3 grid of every task with entries left, one CTA per task.
// Points are taken in walk order (level 0, then the new points of level 1, 2, ...)
// in chunks of kRadThreads. Per chunk, thread t evaluates point f0 + t once for all
// potentials and orders still needed (w U_p, F^A_l, F^B_l, r^N into shared memory);
// then every thread advances the entries it owns over the chunk's points, in the
// reference's order and association, applying libgrpp's per-level rules
// (radial_type2_integral.c:285-315) when an entry passes the last point of a level:
//   level 0: continue; forced refinement while |S|/|estimate| < 1e-3 (estimate valid);
//   converged when |S_L - S_{L-1}| <= 1e-16; otherwise S_prev = S_L, S = S_L / 2.
// An entry therefore ends with exactly the sum the level-by-level walk gives it.
// The walk of a task stops at the first chunk boundary after which no entry is active;
// points evaluated past that are never added. The orders, powers and potentials
// evaluated per point shrink with the set of active entries.
#ifndef GRPP_NO_RADIAL_TABLE_KERNELS
// F_l(r) of every (shell, centre) pair of the batch at every point of the nested grid, one
// CTA per pair and chunk of 128 points: the same point, distance CS (as load_task forms it),
// primitives, exact-zero skips and Bessel rows as the walk's own evaluation, so every order
// l holds the walk's value. Dynamic shared memory: (max fp_lmax + 1) x kRadRow doubles.
__global__ void __launch_bounds__(kRadThreads) ftab_kernel(RadialArgs a, double *ftab)
{
    extern __shared__ double cf[];
    const int tid = threadIdx.x;
    const int nchunk = (kRadGridPts + kRadThreads - 1) / kRadThreads;
    for (int64_t blk = blockIdx.x; blk < (int64_t)a.n_fpairs * nchunk; blk += gridDim.x) {
        const int pr = (int)(blk / nchunk), f = (int)(blk % nchunk) * kRadThreads + tid;
        if (f >= kRadGridPts) continue;
        const int s = a.fp_shell[pr], c = a.fp_centre[pr], lmax = a.fp_lmax[pr];
        const double *So = a.shell_origin + 3 * s, *Co = a.centre_origin + 3 * c;
        double CSv[3];
        for (int d = 0; d < 3; d++) CSv[d] = Co[d] - So[d];
        const double CS2 = CSv[0] * CSv[0] + CSv[1] * CSv[1] + CSv[2] * CSv[2];
        const double CS = sqrt(CS2);
        int lev, i, nr;
        walk_point(f, lev, i, nr);
        double r, w;
        grid_point(f, i, nr, r, w);
        for (int l = 0; l <= lmax; l++) cf[l * kRadRow + tid] = 0.0;
        const double d2 = (r - CS) * (r - CS);
        const int np = a.rp_n[s], off = a.rp_off[s];
#pragma unroll 1
        for (int q = 0; q < np; q++) {
            const double x = a.rp_alpha[off + q];
            const double e = a.rp_coef[off + q] * exp_rn(-x * d2);
            if (e != 0.0) bessel_row_acc(lmax, (2.0 * x * CS) * r, e, cf + tid, kRadRow);
        }
        double *dst = ftab + a.fp_off[pr] + f;
        for (int l = 0; l <= lmax; l++) dst[(int64_t)l * kRadGridPts] = cf[l * kRadRow + tid];
    }
}

// w U_p(r) = w sum_k c_k r^(n_k-2) exp(-zeta_k r^2) at every point of the nested grid, for
// every semilocal potential slot of every GRPP: the grid does not depend on the task, so
// the walk reads these values instead of evaluating the terms for each task. Same point,
// weight, terms, order and exact-zero skips as the walk's own evaluation.
__global__ void wu_table_kernel(RadialArgs a, int n_grpps, double *wu)
{
    const int64_t total = (int64_t)n_grpps * a.wu_npot * kRadGridPts;
    for (int64_t id = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; id < total; id += (int64_t)gridDim.x * blockDim.x) {
        const int f = (int)(id % kRadGridPts);
        const int64_t gp = id / kRadGridPts;
        const int pp = (int)(gp % a.wu_npot), g = (int)(gp / a.wu_npot);
        if (pp >= a.grpp_sl_n[g]) {
            wu[id] = 0.0;
            continue;
        }
        const int pot = a.sl_pot[a.grpp_sl_off[g] + pp];
        int lev, i, nr;
        walk_point(f, lev, i, nr);
        double r, w;
        grid_point(f, i, nr, r, w);
        const double r2 = r * r, ir = 1.0 / r, ir2 = 1.0 / r2;
        double u = 0.0;
        for (int k = 0; k < a.pot_nprim[pot]; k++) {
            const int o = a.pot_prim_off[pot] + k;
            const double ex = exp_rn(-a.pot_alpha[o] * r2);
            if (ex == 0.0) continue;  // the term adds an exact zero
            const double rp = grid_rpow_m2(f, a.pot_powers[o], ir, ir2);  // r^(n-2)
            u += a.pot_coef[o] * rp * ex;
        }
        wu[id] = w * u;
    }
}
#endif  // GRPP_NO_RADIAL_TABLE_KERNELS

#ifndef GRPP_RADIAL_TABLES_ONLY
__global__ void __launch_bounds__(kRadThreads, 5) radial_walk_kernel(RadialArgs a)
{
    __shared__ RadialShared sh;
    __shared__ int s_need[2][4];  // per buffer: max l1, max l2, max N of active entries, potential mask
    __shared__ int s_lvl;         // deepest level at which an entry converged
    extern __shared__ double chunk[];  // [npot + l1max+1 + l2max+1 + dn][kRadRow]
    __shared__ int s_item;
    __shared__ int s_cnt[2];      // lengths of the two active-entry lists
    const int tid = threadIdx.x, lane = tid & 31;
    const bool use_list = a.list_max > 0;
    uint16_t *lists[2] = {reinterpret_cast<uint16_t *>(chunk + a.chunk_doubles),
                          reinterpret_cast<uint16_t *>(chunk + a.chunk_doubles) + a.list_max};
    int next_static = blockIdx.x;
    for (;;) {
        int item;
        if (a.order) {
            // work queue: one pop per CTA (every loop iteration below ends with a barrier)
            __syncthreads();
            if (tid == 0) {
                const int k = atomicAdd(a.queue, 1);
                s_item = k < *a.n_order ? a.order[k] : -1;
            }
            __syncthreads();
            item = s_item;
            if (item < 0) break;
        } else {
            item = next_static;
            next_static += gridDim.x;
            if (item >= a.n_items) break;
            if (!a.walk[item]) continue;
        }
        __syncthreads();
        if (tid < 8) s_need[tid >> 2][tid & 3] = tid == 3 || tid == 7 ? 0 : -1;
        if (tid == 0) {
            s_lvl = 0;
            s_cnt[0] = 0;
        }
        load_task(a, item, sh, tid, kRadThreads);
        const int64_t qo = a.q_off[item];
        double *Q = a.Q + qo, *Sp = a.S_prev + qo;
        const double *SC = a.scr + qo;
        uint8_t *EF = a.eflag + qo;
        const int nE = sh.n_entries, np_a = sh.np_a, np_b = sh.np_b;
        const int npot = sh.npot, l1m = sh.l1max_all, l2m = sh.l2max_all, dn = sh.d_n;
        double *cwu = chunk;                       // [npot][kRadRow]
        double *cf1 = cwu + npot * kRadRow;        // [l1m+1][kRadRow]
        double *cf2 = cf1 + (l1m + 1) * kRadRow;   // [l2m+1][kRadRow]
        double *crn = cf2 + (l2m + 1) * kRadRow;   // [dn][kRadRow]
        const long long t0 = clock64();
        unsigned long long c_acc = 0;
        // what the entries active after screening need from each point
        {
            int n1 = -1, n2 = -1, nN = -1, mask = 0;
            for (int e = tid; e < nE; e += kRadThreads)
                if (EF[e] & kEntActive) {
                    int p, l1, l2, N;
                    decode_entry(sh, e, p, l1, l2, N);
                    n1 = max(n1, l1);
                    n2 = max(n2, l2);
                    nN = max(nN, N);
                    mask |= 1 << p;
                    if (use_list) lists[0][atomicAdd(&s_cnt[0], 1)] = (uint16_t)e;
                }
            atomicMax(&s_need[1][0], n1);
            atomicMax(&s_need[1][1], n2);
            atomicMax(&s_need[1][2], nN);
            atomicOr(&s_need[1][3], mask);
        }
        int any = 1, chunk_no = 0;
        for (int f0 = 0; f0 < kRadGridPts; f0 += kRadThreads, chunk_no++) {
            const int np = min(kRadThreads, kRadGridPts - f0);
            any = __syncthreads_or(any);
            if (!any) break;
            const int nb = (chunk_no + 1) & 1;  // buffer written by the previous chunk (the scan for chunk 0)
            const int u1 = s_need[nb][0], u2 = s_need[nb][1], uN = s_need[nb][2], umask = s_need[nb][3];
            // this chunk's buffer: nobody reads or writes it between the two barriers
            if (tid < 4) s_need[chunk_no & 1][tid] = tid == 3 ? 0 : -1;
            // the list this chunk writes (read last by the chunk before the previous one)
            if (tid == 0) s_cnt[(chunk_no + 1) & 1] = 0;
            if (tid < np) {
                int lev, i, nr;
                walk_point(f0 + tid, lev, i, nr);
                double r, w;
                grid_point(f0 + tid, i, nr, r, w);
                const double r2 = r * r, ir = 1.0 / r, ir2 = 1.0 / r2;
                const double *wug = a.wu ? a.wu + (int64_t)sh.grpp * a.wu_npot * kRadGridPts + f0 + tid : nullptr;
                for (int pp = 0; pp < npot; pp++) {
                    if (!((umask >> pp) & 1)) continue;
                    if (wug) {
                        cwu[pp * kRadRow + tid] = __ldg(wug + (int64_t)pp * kRadGridPts);
                        continue;
                    }
                    double u = 0.0;
                    for (int k = 0; k < sh.pn[pp]; k++) {
                        const int tk = sh.poff[pp] + k;
                        const double ex = exp_rn(-sh.talpha[tk] * r2);
                        if (ex == 0.0) continue;  // the term adds an exact zero
                        const double rp = grid_rpow_m2(f0 + tid, sh.tpow[tk], ir, ir2);  // r^(n-2)
                        u += sh.tcoef[tk] * rp * ex;
                    }
                    cwu[pp * kRadRow + tid] = w * u;
                }
                if (a.ftab) {
                    // F^A_l, F^B_l of this point from the (shell, centre) tables
                    const double *FA = a.ftab + sh.fa_off + f0 + tid, *FB = a.ftab + sh.fb_off + f0 + tid;
                    for (int l = 0; l <= u1; l++) cf1[l * kRadRow + tid] = __ldg(FA + (int64_t)l * kRadGridPts);
                    for (int l = 0; l <= u2; l++) cf2[l * kRadRow + tid] = __ldg(FB + (int64_t)l * kRadGridPts);
                } else {
                    for (int l = 0; l <= u1; l++) cf1[l * kRadRow + tid] = 0.0;
                    for (int l = 0; l <= u2; l++) cf2[l * kRadRow + tid] = 0.0;
                }
                const double dA2 = (r - sh.CA) * (r - sh.CA), dB2 = (r - sh.CB) * (r - sh.CB);
                if (!a.ftab && u1 >= 0) {
#pragma unroll 1
                    for (int q = 0; q < np_a; q++) {
                        const double e = sh.ca[q] * exp_rn(-sh.xa[q] * dA2);
                        if (e != 0.0) bessel_row_acc(u1, sh.ka[q] * r, e, cf1 + tid, kRadRow);
                    }
                }
                if (!a.ftab && u2 >= 0) {
#pragma unroll 1
                    for (int q = 0; q < np_b; q++) {
                        const double e = sh.cb[q] * exp_rn(-sh.xb[q] * dB2);
                        if (e != 0.0) bessel_row_acc(u2, sh.kb[q] * r, e, cf2 + tid, kRadRow);
                    }
                }
                if (c_tab.grid) {
                    // r^N = pow(r, N) as libgrpp tabulates it (radial_type2_integral.c:440-441)
                    const double *gp = c_tab.grid + (size_t)kGridRowPow0 * kGridPts + f0 + tid;
                    for (int n = 0; n <= uN; n++) crn[n * kRadRow + tid] = __ldg(gp + (size_t)n * kGridPts);
                } else {
                    double rn = 1.0;
                    for (int n = 0; n <= uN; n++) {
                        crn[n * kRadRow + tid] = rn;
                        rn *= r;
                    }
                }
            }
            __syncthreads();
            int lev0, i0, nr0;
            walk_point(f0, lev0, i0, nr0);
            int my_active = 0, n1 = -1, n2 = -1, nN = -1, mask = 0, my_lvl = 0;
            // active entries: from the compacted list (an even share per thread), else all entries
            const int ncur = use_list ? s_cnt[chunk_no & 1] : nE;
            const uint16_t *lcur = lists[chunk_no & 1];
            uint16_t *lnext = lists[(chunk_no + 1) & 1];
            for (int k = tid; k < ncur; k += kRadThreads) {
                const int e = use_list ? lcur[k] : k;
                uint8_t fl = EF[e];
                if (!(fl & kEntActive)) continue;
                int p, l1, l2, N;
                decode_entry(sh, e, p, l1, l2, N);
                const double *pwu = cwu + p * kRadRow, *p1 = cf1 + l1 * kRadRow, *p2 = cf2 + l2 * kRadRow,
                             *pn = crn + N * kRadRow;
                double s = Q[e], sp = Sp[e];
                int q = 0, L = lev0;
                while (q < np) {
                    const int lend = level_last_point(L);
                    const int qe = min(np, lend - f0 + 1);
                    for (; q < qe; q++) s = __dadd_rn(s, __dmul_rn(__dmul_rn(__dmul_rn(pwu[q], p1[q]), p2[q]), pn[q]));
                    if (f0 + qe - 1 != lend) break;  // level continues in the next chunk
                    // end of level L for this entry (radial_type2_integral.c:285-315)
                    const bool forced = L == 0 || ((fl & kEntScrOk) && (fabs(s) / fabs(SC[e]) < 0.001));
                    if (!forced && fabs(s - sp) <= 1e-16) {
                        fl &= ~kEntActive;
                        my_lvl = max(my_lvl, L);
                        break;
                    }
                    if (L < kRadMaxLevel) {
                        sp = s;
                        s = 0.5 * s;
                    }
                    L++;
                }
                c_acc += q;
                Q[e] = s;
                Sp[e] = sp;
                EF[e] = fl;
                if (fl & kEntActive) {
                    if (use_list) lnext[atomicAdd(&s_cnt[(chunk_no + 1) & 1], 1)] = (uint16_t)e;
                    my_active = 1;
                    n1 = max(n1, l1);
                    n2 = max(n2, l2);
                    nN = max(nN, N);
                    mask |= 1 << p;
                }
            }
            if (my_active) {
                atomicMax(&s_need[chunk_no & 1][0], n1);
                atomicMax(&s_need[chunk_no & 1][1], n2);
                atomicMax(&s_need[chunk_no & 1][2], nN);
                atomicOr(&s_need[chunk_no & 1][3], mask);
            }
            if (my_lvl) atomicMax(&s_lvl, my_lvl);
            any = my_active;
        }
        any = __syncthreads_or(any);
        // deepest level walked: the cap if entries are still active, else the last convergence
        const int level_reached = any ? kRadMaxLevel : s_lvl;
        if (tid == 0 && a.stop_level) a.stop_level[item] = (int8_t)level_reached;
        if (tid == 0 && a.pred_level && level_reached > a.pred_level[item] + 1) atomicAdd(a.fallback_count, 1);
        if (a.counters) {
            unsigned long long v = c_acc;
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) atomicAdd(a.counters + kRadCntAccum, v);
            if (tid == 0) {
                // algorithmic work of the shared grid up to the stop level (every point once,
                // every order and potential term at every point)
                const unsigned long long pts = (unsigned long long)((1 << (level_reached + 5)) - 1);
                atomicAdd(a.counters + kRadCntPoints, pts);
                atomicAdd(a.counters + kRadCntBessel, pts * (unsigned long long)(np_a * (l1m + 1) + np_b * (l2m + 1)));
                atomicAdd(a.counters + kRadCntPrimPts, pts * (unsigned long long)(np_a + np_b));
                atomicAdd(a.counters + kRadCntTermPts, pts * (unsigned long long)sh.nterm_tot);
                atomicAdd(a.counters + kRadCntPowPts, pts * (unsigned long long)dn);
                atomicAdd(a.counters + kRadCntQuadCycles, (unsigned long long)(clock64() - t0));
                atomicAdd(a.counters + kRadCntItems, 1ull);
                atomicAdd(a.counters + kRadCntLevels, (unsigned long long)(level_reached + 1));
            }
        }
    }
}

// ---- the walk over tabulated integrands: radial_walk_group_kernel ------------------------------
//
// The same walk (points, per-level rules, sums: radial_walk_kernel above) when w U_p, F_l and r^N
// come from tables. What it does differently:
//  * A thread advances a group of up to kWalkN entries of one (p, l1, l2) whose N differ by 2:
//    ((w U) F1) F2 is formed once per point for the group, and the entries' sums are independent
//    chains: 3 + k shared loads, 2 + k products and k additions for k entries, where each entry took 4
//    loads, 3 products and a dependent addition.
//  * Most points belong to the deep levels of a few entries (63 active entries per point on the s..g
//    workload), so what counts there is the latency of a chunk: the rows that are still needed are
//    packed, and a chunk takes as many points as the block's shared memory holds of them (128 to
//    1024, within one level), copied asynchronously, every row in flight at once.
//  * Chunks start one before libgrpp's first point (a point of weight 0), so that levels 0 to 2 are the
//    first 128 points and every later level starts and ends with a chunk; rows of an odd number of
//    16-byte units, read two points at a time without bank conflicts.
//  * Items are taken by centre, so that the F_l tables of one centre's shells stay in L2; a batch of
//    few items shares the groups of an item between nparts CTAs.
//  * The lists of active groups carry their entries' active bits; flags, previous sums and estimates
//    are read at the ends of levels only.
// Bound by shared-memory loads (75% of the cycles). Walk with its tables and ordering, four blocks
// per SM against five: 26.6 and 26.5 ms on 65536 s..g tasks, 21.3 and 22.5 on a 15-atom molecule,
// where the walk by single entries took 30.0 and 31.8; a 200-task molecule 1.21 -> 0.42 ms.
// Groups of the four order pairs L -+ k1, L -+ k2 (a third of the loads) leave too few threads
// busy: 35.7 ms on the first.
constexpr int kWalkN = 4;
constexpr int kWalkPts = 128;            // points of the smallest chunk
constexpr int kWalkMaxPts = 1024;
constexpr int kWalkRow = kWalkPts + 2;
constexpr int kWalkThreads = 128;
struct WalkGroup {
    uint8_t l1, l2, n0, cnt;  // orders; N = n0, n0 + 2, .., cnt of them
};

struct WalkArgs {
    const WalkGroup *groups;
    const int2 *cls;     // per class (L, la, lb): offset into groups, count
    const int *perm;     // items by potential centre
    int nparts;          // CTAs per item
    int list_max;        // capacity of the active-group lists (groups of one item at most)
    int chunk_doubles;   // doubles of point rows before the lists
    unsigned *item_level;  // nparts > 1: levels that an item's finished parts reached (a bit each) and, from bit 16, how many have finished
};

// 8 bytes from global to shared memory, asynchronously (zero: writes 0)
__device__ __forceinline__ void copy8_async(double *dst, const double *src, bool zero)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(zero ? 0 : 8)
                 : "memory");
}

// The sums of K entries over the point pairs x0..x1-1, each in point order: s += (((w U) F1) F2) r^N.
// Four pairs of points in flight hide the loads behind the additions where a block is alone on its
// SM (one f x d block: call 535 us with two, 512 with four, 509 with eight; 65536 s..g tasks 80.3, 79.0, 79.5 ms).
template <int K>
__device__ __forceinline__ void walk_advance(int x0, int x1, const double2 *pw, const double2 *p1, const double2 *p2,
                                             const double2 *const *pn, double *s)
{
#pragma unroll 4
    for (int x = x0; x < x1; x++) {
        const double2 vw = pw[x], v1 = p1[x], v2 = p2[x];
        const double tx = __dmul_rn(__dmul_rn(vw.x, v1.x), v2.x), ty = __dmul_rn(__dmul_rn(vw.y, v1.y), v2.y);
#pragma unroll
        for (int q = 0; q < K; q++) {
            const double2 vn = pn[q][x];
            s[q] = __dadd_rn(s[q], __dmul_rn(tx, vn.x));
            s[q] = __dadd_rn(s[q], __dmul_rn(ty, vn.y));
        }
    }
}

__global__ void __launch_bounds__(kWalkThreads, 4) radial_walk_group_kernel(RadialArgs a, WalkArgs w)
{
    extern __shared__ __align__(16) double wsm[];
    __shared__ int pL[kRadMaxPots], pent[kRadMaxPots], pgrp[kRadMaxPots], gpre[kRadMaxPots + 1];
    __shared__ int s_need[2][4];  // per buffer: max l1, max l2, max N of active entries, potential mask
    __shared__ int s_cnt[2], s_lvl, s_item, s_part;
    const int tid = threadIdx.x, lane = tid & 31, NT = blockDim.x;
    // active groups: potential << 27 | index within the potential's groups << 4 | active entries
    unsigned *lists[2] = {(unsigned *)(wsm + w.chunk_doubles), (unsigned *)(wsm + w.chunk_doubles) + w.list_max};
    const int n_units = (a.order ? *a.n_order : a.n_items) * w.nparts;
    for (;;) {
        __syncthreads();
        if (tid == 0) {
            int item = -1, part = 0;
            for (;;) {
                const int u = atomicAdd(a.queue, 1);
                if (u >= n_units) break;
                const int k = u / w.nparts;
                const int it = a.order ? a.order[k] : w.perm[k];
                if (!a.order && !a.walk[it]) continue;
                item = it;
                part = u - k * w.nparts;
                break;
            }
            s_item = item;
            s_part = part;
            s_lvl = 0;
            s_cnt[0] = 0;
        }
        if (tid < 8) s_need[tid >> 2][tid & 3] = (tid & 3) == 3 ? 0 : -1;
        __syncthreads();
        const int item = s_item, part = s_part;
        if (item < 0) break;
        const int t = a.item_task[item], c = a.task_c[t], gr = a.centre_grpp[c];
        const int la = a.shell_L[a.task_a[t]], lb = a.shell_L[a.task_b[t]], dn = la + lb + 1, npot = a.grpp_sl_n[gr];
        if (tid < 32) {
            int sz = 0, ng = 0;
            if (tid < npot) {
                const int L = a.pot_L[a.sl_pot[a.grpp_sl_off[gr] + tid]];
                const int2 cl = w.cls[(L * (kMaxL + 1) + la) * (kMaxL + 1) + lb];
                pL[tid] = L;
                pgrp[tid] = cl.x;
                sz = (L + la + 1) * (L + lb + 1) * dn;
                ng = cl.y;
            }
            int es = sz, gs = ng;
            for (int o = 1; o < 32; o <<= 1) {
                const int e = __shfl_up_sync(0xffffffffu, es, o), g = __shfl_up_sync(0xffffffffu, gs, o);
                if (lane >= o) {
                    es += e;
                    gs += g;
                }
            }
            if (tid < npot) {
                pent[tid] = es - sz;
                gpre[tid + 1] = gs;
            }
            if (tid == 0) gpre[0] = 0;
        }
        __syncthreads();
        const int64_t qo = a.q_off[item];
        double *Q = a.Q + qo, *Sp = a.S_prev + qo;
        const double *SC = a.scr + qo;
        uint8_t *EF = a.eflag + qo;
        const long long t0 = clock64();
        unsigned long long c_acc = 0;
        const int G = gpre[npot], glo = (int)((int64_t)G * part / w.nparts), ghi = (int)((int64_t)G * (part + 1) / w.nparts);
        {  // groups with an entry left by the screening, and what they need of each point
            int n1 = -1, n2 = -1, nN = -1, mask = 0;
            for (int gb = glo + (tid & ~31); gb < ghi; gb += NT) {
                const int g = gb + lane;
                int p = 0, loc = 0;
                unsigned on = 0;
                WalkGroup W{};
                if (g < ghi) {
                    while (gpre[p + 1] <= g) p++;
                    loc = g - gpre[p];
                    W = w.groups[pgrp[p] + loc];
                    const uint8_t *E = EF + pent[p] + (W.l1 * (pL[p] + lb + 1) + W.l2) * dn + W.n0;
                    for (int q = 0; q < W.cnt; q++)
                        if (E[2 * q] & kEntActive) on |= 1u << q;
                }
                const unsigned keep = __ballot_sync(0xffffffffu, on != 0);
                int at = 0;
                if (lane == 0 && keep) at = atomicAdd(&s_cnt[0], __popc(keep));
                at = __shfl_sync(0xffffffffu, at, 0);
                if (!on) continue;
                lists[0][at + __popc(keep & ((1u << lane) - 1))] = (unsigned)p << 27 | (unsigned)loc << 4 | on;
                n1 = max(n1, (int)W.l1);
                n2 = max(n2, (int)W.l2);
                nN = max(nN, W.n0 + 2 * (W.cnt - 1));
                mask |= 1 << p;
            }
            if (mask) {
                atomicMax(&s_need[1][0], n1);
                atomicMax(&s_need[1][1], n2);
                atomicMax(&s_need[1][2], nN);
                atomicOr(&s_need[1][3], mask);
            }
        }
        __syncthreads();
        const double *FA = a.ftab + a.fp_off[a.item_fa[item]], *FB = a.ftab + a.fp_off[a.item_fb[item]];
        const double *wug = a.wu + (int64_t)gr * a.wu_npot * kRadGridPts;
        const double *rng = c_tab.grid + (size_t)kGridRowPow0 * kGridPts;
        int any = 0;
        for (int q0 = 0, npts = 0, cur = 0; q0 <= kRadGridPts; q0 += npts, cur ^= 1) {
            const int nb = cur ^ 1, ncur = s_cnt[cur];
            any = ncur > 0;
            if (!any) break;
            const int u1 = s_need[nb][0], u2 = s_need[nb][1], uN = s_need[nb][2], umask = s_need[nb][3];
            // what this chunk refills: nobody reads it before the next barrier
            if (tid < 4) s_need[cur][tid] = tid == 3 ? 0 : -1;
            if (tid == 0) s_cnt[nb] = 0;
            // ---- the chunk: points q0 .. q0 + npts - 1 of one level (levels 0..2 for q0 = 0), column x
            // being walk-order point q0 + x - 1
            const int nw = __popc(umask), rows = nw + u1 + u2 + uN + 3;
            npts = kWalkPts;
            if (q0 > 0) {
                const int left = (2 << (31 - __clz(q0))) - q0;  // points to the end of the level
                while (2 * npts <= min(left, kWalkMaxPts) && rows * (2 * npts + 2) <= w.chunk_doubles) npts *= 2;
            }
            const int rst = npts + 2;
            double *cf1 = wsm + nw * rst, *cf2 = cf1 + (u1 + 1) * rst, *crn = cf2 + (u2 + 1) * rst;
            for (int x = tid; x < npts; x += NT) {
                const int f = max(q0 + x - 1, 0);
                const bool dummy = q0 + x == 0;
                double *d = wsm + x;
                for (int m = umask; m; m &= m - 1, d += rst)
                    copy8_async(d, wug + (int64_t)(__ffs(m) - 1) * kRadGridPts + f, dummy);
                for (int l = 0; l <= u1; l++, d += rst) copy8_async(d, FA + (int64_t)l * kRadGridPts + f, false);
                for (int l = 0; l <= u2; l++, d += rst) copy8_async(d, FB + (int64_t)l * kRadGridPts + f, false);
                for (int n = 0; n <= uN; n++, d += rst) copy8_async(d, rng + (size_t)n * kGridPts + f, false);
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            // level that ends with this chunk (q0 = 0: levels 0..2): -1 if none
            const int qe = q0 + npts, lend = (qe & (qe - 1)) == 0 ? 31 - __clz(qe) - 5 : -1;
            int n1 = -1, n2 = -1, nN = -1, mask = 0, my_lvl = 0;
            for (int k0 = tid & ~31; k0 < ncur; k0 += NT) {
                // a warp's lanes run together: the list keeps groups of equal size side by side
                const bool have = k0 + lane < ncur;
                const unsigned id = lists[cur][have ? k0 + lane : k0];
                const int p = id >> 27;
                const WalkGroup W = w.groups[pgrp[p] + ((id >> 4) & 0x7fffff)];
                unsigned act = have ? id & 15u : 0u;
                const int e0 = pent[p] + (W.l1 * (pL[p] + lb + 1) + W.l2) * dn + W.n0;
                double sm[kWalkN];
                const double2 *pw = (const double2 *)(wsm + __popc(umask & ((1 << p) - 1)) * rst),
                              *p1 = (const double2 *)(cf1 + W.l1 * rst), *p2 = (const double2 *)(cf2 + W.l2 * rst), *pn[kWalkN];
#pragma unroll
                for (int q = 0; q < kWalkN; q++) {
                    const bool on = (act >> q) & 1u;
                    sm[q] = on ? Q[e0 + 2 * q] : 0.0;
                    // an entry that is not active takes a row that is there; its sum is not stored
                    pn[q] = (const double2 *)(crn + (on ? W.n0 + 2 * q : 0) * rst);
                }
                int x = 0;
                for (int seg = 0; seg < 3; seg++) {
                    // q0 = 0: levels 0, 1, 2 end after 32, 64, 128 points; else the whole chunk
                    const int xe = q0 == 0 ? 16 << seg : npts / 2;
                    c_acc += (unsigned)(2 * (xe - x) - (q0 + x == 0)) * __popc(act);
                    const int K = __reduce_max_sync(0xffffffffu, 32 - __clz(act));  // of the warp's largest group
                    if (K == 4) walk_advance<4>(x, xe, pw, p1, p2, pn, sm);
                    else if (K == 3) walk_advance<3>(x, xe, pw, p1, p2, pn, sm);
                    else if (K == 2) walk_advance<2>(x, xe, pw, p1, p2, pn, sm);
                    else if (K == 1) walk_advance<1>(x, xe, pw, p1, p2, pn, sm);
                    x = xe;
                    const int L = q0 == 0 ? seg : lend;
                    if (L >= 0) {
                        // end of level L (radial_type2_integral.c:285-315); an entry that has converged
                        // keeps its sum
#pragma unroll
                        for (int q = 0; q < kWalkN; q++)
                            if ((act >> q) & 1u) {
                                const int en = e0 + 2 * q;
                                bool conv = false;
                                if (L > 0) {
                                    const bool forced = (EF[en] & kEntScrOk) && (fabs(sm[q]) / fabs(SC[en]) < 0.001);
                                    conv = !forced && fabs(sm[q] - Sp[en]) <= 1e-16;
                                }
                                if (conv) {
                                    act &= ~(1u << q);
                                    Q[en] = sm[q];
                                    EF[en] &= (uint8_t)~kEntActive;
                                    my_lvl = max(my_lvl, L);
                                } else if (L < kRadMaxLevel) {
                                    Sp[en] = sm[q];
                                    sm[q] = 0.5 * sm[q];
                                }
                            }
                    }
                    if (q0 > 0) break;
                }
#pragma unroll
                for (int q = 0; q < kWalkN; q++)
                    if ((act >> q) & 1u) Q[e0 + 2 * q] = sm[q];
                const unsigned keep = __ballot_sync(0xffffffffu, act != 0);
                int at = 0;
                if (lane == 0 && keep) at = atomicAdd(&s_cnt[nb], __popc(keep));
                at = __shfl_sync(0xffffffffu, at, 0);
                if (act) {
                    lists[nb][at + __popc(keep & ((1u << lane) - 1))] = (id & ~15u) | act;
                    n1 = max(n1, (int)W.l1);
                    n2 = max(n2, (int)W.l2);
                    nN = max(nN, W.n0 + 2 * (31 - __clz(act)));
                    mask |= 1 << p;
                }
            }
            if (mask) {
                atomicMax(&s_need[cur][0], n1);
                atomicMax(&s_need[cur][1], n2);
                atomicMax(&s_need[cur][2], nN);
                atomicOr(&s_need[cur][3], mask);
            }
            if (my_lvl) atomicMax(&s_lvl, my_lvl);
            __syncthreads();  // the next list and needs are complete; the rows are consumed
        }
        if (a.counters) {
            unsigned long long v = c_acc;
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) atomicAdd(a.counters + kRadCntAccum, v);
            if (tid == 0) atomicAdd(a.counters + kRadCntQuadCycles, (unsigned long long)(clock64() - t0));
        }
        if (tid == 0) {
            // deepest level walked: the cap if the last chunk was walked, else the last convergence; the
            // item's is known to the CTA that finishes its last part
            int level_reached = any ? kRadMaxLevel : s_lvl;
            bool last = true;
            if (w.nparts > 1) {
                atomicOr(w.item_level + item, 1u << level_reached);
                const unsigned v = atomicAdd(w.item_level + item, 1u << 16);
                last = (int)(v >> 16) == w.nparts - 1;
                level_reached = 31 - __clz(v & 0xffffu);
            }
            if (last && a.stop_level) a.stop_level[item] = (int8_t)level_reached;
            if (last && a.pred_level && level_reached > a.pred_level[item] + 1) atomicAdd(a.fallback_count, 1);
            if (last && a.counters) {
                // algorithmic work of the shared grid up to the stop level (every point once,
                // every order and potential term at every point)
                const unsigned long long pts = (unsigned long long)((1 << (level_reached + 5)) - 1);
                const int np_a = a.rp_n[a.task_a[t]], np_b = a.rp_n[a.task_b[t]];
                int terms = 0, l1m = 0, l2m = 0;
                for (int p = 0; p < npot; p++) {
                    terms += a.pot_nprim[a.sl_pot[a.grpp_sl_off[gr] + p]];
                    l1m = max(l1m, pL[p] + la);
                    l2m = max(l2m, pL[p] + lb);
                }
                atomicAdd(a.counters + kRadCntPoints, pts);
                atomicAdd(a.counters + kRadCntBessel, pts * (unsigned long long)(np_a * (l1m + 1) + np_b * (l2m + 1)));
                atomicAdd(a.counters + kRadCntPrimPts, pts * (unsigned long long)(np_a + np_b));
                atomicAdd(a.counters + kRadCntTermPts, pts * (unsigned long long)terms);
                atomicAdd(a.counters + kRadCntPowPts, pts * (unsigned long long)dn);
                atomicAdd(a.counters + kRadCntItems, 1ull);
                atomicAdd(a.counters + kRadCntLevels, (unsigned long long)(level_reached + 1));
            }
        }
    }
}
#endif  // GRPP_RADIAL_TABLES_ONLY

}  // namespace grpp

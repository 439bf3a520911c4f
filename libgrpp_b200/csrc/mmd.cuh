// Type 1 (radially local) GRPP integrals by McMurchie-Davidson, and two-centre overlaps by
// Obara-Saika, one thread block per work item.
//
// Reference algorithm: libgrpp/type1_mcmurchie_davidson.c:107-622 and
// libgrpp/type1_integrals.c:43-78 (sum over potential terms k of c_k times the
// primitive-pair contraction), libgrpp/overlap.c:39-139.
//
// A work item is <bra| c r^(n-2) exp(-zeta r^2) (centred at C) |ket> summed over the terms of
// one potential, or the overlap <bra|ket>. For a primitive triple (i, j, k) with exponents
// a, b, zeta, q = a + b + zeta, Q = (a A + b B + zeta C) / q and K_d the Gaussian product
// factor of axis d:
//   n = 2, and the overlap (zeta = 0):  (pi/q)^(3/2) prod_d S_d[i_d][j_d], Obara-Saika tables;
//   n = 1, n = 0:                       sum_tuv E^x_t E^y_u E^z_v R^0_tuv,
// E[axis][i][j][t] the Hermite expansion coefficients and R^n_tuv the auxiliary integrals, by
// levels s = t + u + v (level s from s-1 and s-2) from (-2q)^n F_n (Boys) for n = 1 and from
// (2q)^n G_n for n = 0. The n = 0 levels are differences R^(n+1) - 2q R^n that cancel for tight
// exponents far from C; G_n, the powers of 2q and the levels therefore keep libgrpp's operations
// one by one, so that the lost digits are the same ones.
//
// Mapping. A block takes the item's triples in groups of up to 64, for which it forms scalars
// (a thread per triple and axis) and auxiliary values (four threads per triple), and these in
// batches of T (a power of two per (la, lb) and kind, MmdClass). Every phase of a batch runs
// over (entry, triple) pairs with the triple fastest: tables are laid out [entry][T], so the
// lanes of a warp work on few different entries, addresses are consecutive and the update
// programs (which entry comes from which) are read once per T triples. Per batch: step
// s = 1..S does the E wavefront i + j = s and the R level s together (one barrier each), then
// X[t,u][az,bz] = sum_v E^z_v R^0_tuv and, per Cartesian pair, sum_t E^x_t sum_u E^y_u X.
// Splitting the contraction at z makes it about 4 operations per pair where the triple sum
// needs 14 (g x g) to 60 (i x i).
// The sums of an item are formed in parts that the item alone fixes (mmd_part_size), so that they do not depend
// on how many blocks take it.
// Triples whose Gaussian product exponents sum to more than 800 are dropped: K_x K_y K_z < 1e-347
// there, so their contributions underflow.
//
// What bounds it: shared-memory latency between the barriers of the S steps (FP64 is mostly
// idle). Three blocks of 256 threads per SM with 70 kB each (T as large as fits) measured faster
// than two with 104 kB (11.6 ms), four with 52 kB (10.3) or one with 204 kB (20.0) on the 65536
// tasks of the s..g workload: 10.0 ms, against 40.7 ms for one warp per item walking its triples
// one by one. The matrices of a 15-atom molecule with i shells, whose largest class set the registers
// and shared memory of every item there: 51.9 -> 6.6 ms; a 200-task molecule: 2.0 -> 0.19 ms.
#pragma once

#include "grpp_common.cuh"
#include "specfunc.cuh"
#include "radial.cuh"  // RadialCounter slots shared with the type 1 kernel

namespace grpp {

struct MmdItem {
    int bra, ket;        // shell indices
    int ket_at_centre;   // 1: ket origin is the centre C (outercore shells)
    int centre;          // centre index (origin of the potential)
    int pot;             // potential index, or -1 for an overlap
    int out_kind;        // 0: arep output, 1: outercore U scratch, 2: outercore S scratch
    int64_t out_off;     // offset of the nbra x nket row-major block
    int pairs;           // offset of the item's Cartesian pair table (MmdArgs::pairs)
    int cls;             // class index la * kMmdCls + lb
};

constexpr int kMmdThreads = 256;
constexpr int kMmdMaxL = 8;               // largest angular momentum whose tables are built
constexpr int kMmdCls = kMmdMaxL + 1;
constexpr int kMmdMaxPrims = 64;          // primitives per shell (the engine's limit)
constexpr int kMmdMaxLgT = 6;
constexpr int kMmdMaxParts = 32;          // parts of one item's triples, each with a sum of its own
constexpr int kMmdMaxShares = 16;         // blocks that share one item's parts
constexpr int kMmdSmem = 70 * 1024;       // dynamic shared memory at most: three blocks per SM
constexpr int kMmdGroup = 64;             // triples whose scalars and auxiliary values are formed together
constexpr int kMmdRing = 512;             // live triples waiting: at most kMmdGroup - 1 + kMmdThreads
constexpr double kMmdDropArg = 800.0;     // sum of the Gaussian product exponents that underflows
constexpr double kPi15 = 5.568327996831708;  // pi^(3/2), correctly rounded
static_assert(4 * kMmdGroup == kMmdThreads && (1 << kMmdMaxLgT) <= kMmdGroup, "four threads per triple of a group");

// Tables of one (la, lb), built once per device (mmd_build_classes)
struct MmdClass {
    int la, lb, S;
    int nE;              // Hermite coefficients of the three axes, [ax][(i, j)][t <= i + j]
    int nR0;             // R^0_tuv, rows (t, u) of consecutive v
    int nX;              // X[(az, bz)][t][u], t + u <= S - az - bz
    int maxlev;          // largest level of R^n_tuv
    int e_off, o_off, z_off, r_off;  // programs: E, Obara-Saika, X, R
    int lv;              // level starts in MmdArgs::levels: S + 2 each of E, Obara-Saika, R
    int lgT[2];          // log2 of the triples per batch: [0] n = 2 and overlap, [1] n = 0, 1
};

struct MmdArgs {
    const MmdItem *items;
    int n_items;
    const int *shell_nprim, *shell_prim_off, *shell_L;
    const double *prim_coef, *prim_alpha, *shell_origin;
    const int *pot_nprim, *pot_prim_off, *pot_powers;
    const double *pot_coef, *pot_alpha;
    const int *pot_perm, *pot_n2;  // per potential: term order with the n = 2 terms first, their number
    const double *centre_origin;
    double *out[3];
    unsigned long long *counters;  // kRadCntMmdTriples / kRadCntMmdFlops slots (may be null)
    const MmdClass *classes;
    const int *levels;
    // update programs, one int2 per entry (mmd_e_code, mmd_o_code, mmd_r_code, mmd_z_code)
    const int2 *etab, *otab, *rtab, *ztab;
    // per class of (bra, ket) Cartesian tables, one int4 per pair (mmd_pair)
    const int4 *pairs;
    // dynamic schedule: blocks pop positions from *queue (zeroed before the launch) and take
    // units[position]; the host orders them by decreasing estimated work. A unit is an item or, in
    // small batches, one of up to kMmdMaxShares shares of its parts (below): x item, y share |
    // number of shares << 8, z offset of the item's partial sums in part_out, w its counter in
    // part_cnt (zeroed before the launch)
    const int4 *units;
    int n_units;
    int *queue;
    double *part_out;
    int *part_cnt;
};

__host__ __device__ inline int mmd_tet(int m) { return (m + 1) * (m + 2) * (m + 3) / 6; }
// first t of E[ax][i][j] among the axis' coefficients
__host__ __device__ inline int mmd_e_row(int lb, int i, int j)
{
    const int lb1 = lb + 1;
    return lb1 * i * (i - 1) / 2 + i * (lb1 * (lb1 + 1) / 2) + j * i + j * (j + 1) / 2;
}
__host__ __device__ inline int mmd_e_axis(int la, int lb) { return (la + 1) * (lb + 1) * (la + lb + 2) / 2; }
// start of row (t, u) in the R^0 layout: rows ordered t-major, then u
__host__ __device__ __forceinline__ int r0_row(int S, int t, int u)
{
    return mmd_tet(S) - mmd_tet(S - t) + u * (S - t + 1) - u * (u - 1) / 2;
}
// index of (u + v = k, v) within level s
__host__ __device__ __forceinline__ int r_in_level(int u, int v) { return (u + v) * (u + v + 1) / 2 + v; }

// Triples per part of an item with n triples (all terms): a group, half of one where a batch of the class
// has at most 8 triples (high l, few triples that take long), or as many of these as make at most
// kMmdMaxParts parts (the two kinds of terms apart). The sums of the parts are added in order, so that an
// item has the same bits whether one block takes all of its parts or several share them. Twice the size left
// shares of molecules with i shells uneven (2.65 against 2.5 ms for five atoms); half of it gained nothing.
__host__ __device__ inline int mmd_part_size(int64_t n, int lgT)
{
    const int unit = lgT <= 3 ? kMmdGroup / 2 : kMmdGroup;
    return unit * (int)((n / unit + 2) / (kMmdMaxParts - 1) + 1);
}

// doubles of shared memory: per triple of a group (scalars and R^n_000), and of a batch (tables)
__host__ __device__ inline int mmd_group_doubles(const MmdClass &c) { return 15 + c.S + 1; }
__host__ __device__ inline int mmd_batch_doubles(const MmdClass &c, int kind)
{
    if (kind == 0) return 3 * (c.la + 1) * (c.lb + 1);
    const int u = c.nX > 3 * c.maxlev ? c.nX : 3 * c.maxlev;
    return c.nE + c.nR0 + u;
}
// sums of the Cartesian pairs: one per 32 triples of a batch
__host__ __device__ inline int mmd_sum_groups(const MmdClass &c)
{
    const int lg = c.lgT[0] > c.lgT[1] ? c.lgT[0] : c.lgT[1];
    return lg > 5 ? 1 << (lg - 5) : 1;
}
__host__ __device__ inline int mmd_smem_doubles(const MmdClass &c)
{
    const int a = mmd_batch_doubles(c, 0) << c.lgT[0], b = mmd_batch_doubles(c, 1) << c.lgT[1];
    return ncart(c.la) * ncart(c.lb) * mmd_sum_groups(c) + mmd_group_doubles(c) * kMmdGroup + (a > b ? a : b);
}

// ---- update programs (host-built)
// Hermite coefficient (type1_mcmurchie_davidson.c:569-622), t = 0:
//   P E[src] + (second ? E[src + 1] : 0), P = (Q-A)[ax] or (Q-B)[ax] (side 1)
// t >= 1: (i E[src1] + j E[src2]) / (2 q t)
inline int2 mmd_e_code0(int dst, int src, int ax, int side, bool second)
{
    return int2{dst | (src << 13) | (1 << 30), (ax << 13) | (side << 20) | ((second ? 1 : 0) << 24)};
}
inline int2 mmd_e_code(int dst, int src1, int src2, int ax, int i, int j, int t)
{
    return int2{dst | (src1 << 13), src2 | (ax << 13) | (t << 15) | (i << 20) | (j << 24)};
}
// Obara-Saika table (overlap.c:92-120): P S[s1] + (n2 S[s2] + n3 S[s3]) / (2q)
inline int2 mmd_o_code(int dst, int s1, int s2, int s3, int n2, int n3, int ax, int side)
{
    return int2{dst | (s1 << 10) | (s2 << 20), s3 | (n2 << 10) | (n3 << 14) | (ax << 18) | (side << 20)};
}
// R^n_tuv at level s (type1_mcmurchie_davidson.c:457-564): (k - 1) D2 + (Q-C)[ax] D1 with
// D1 = prev1[src1 + ne1] (- 2q prev1[src1] for the 1/r^2 terms), D2 likewise from prev2 (k > 1)
inline int2 mmd_r_code(int src1, int src2, int dst_r0, int k, int ax)
{
    return int2{src1 | (src2 << 16), dst_r0 | (k << 14) | (ax << 19)};
}
constexpr int kMmdNoR0 = 8191;  // order n > 0: not an R^0 value
// X entry: sum_{v <= vz} E[zrow + v] R0[row + v]
inline int2 mmd_z_code(int row, int zrow, int vz) { return int2{row | (zrow << 16), vz}; }
// Cartesian pair: E rows of axes x and y; start of its X rows, their count W + 1 and tx, uy; the
// three Obara-Saika entries; index in the output block
inline int4 mmd_pair(int ex, int ey, int xbase, int W, int tx, int uy, int o0, int o1, int o2, int out)
{
    return int4{ex | (ey << 16), xbase | (W << 16) | (tx << 21) | (uy << 26), o0 | (o1 << 10) | (o2 << 20), out};
}

// FP64 operations of one primitive triple of libgrpp's algorithm, by phase (FMA = 2, exp/div/sqrt/pow
// = 1), for the counting build: setup 40; a Hermite coefficient 5; an auxiliary function value
// 16 (Boys, 6th-order Taylor) or 100 per G_n series; an R^n_tuv entry 5; a term
// E_x E_y E_z R of the contraction 3, plus 3 per Cartesian pair.
__host__ __device__ inline unsigned long long mmd_e_count(int la, int lb)
{
    return 3ull * ((la + 1) * (lb + 1) + (lb + 1) * la * (la + 1) / 2 + (la + 1) * lb * (lb + 1) / 2);
}
__host__ __device__ inline int mmd_r_size(int smax)
{
    // sum over levels s of (s+1)(s+2)/2 entries x (smax-s+1) orders
    int tot = 0;
    for (int s = 0; s <= smax; s++) tot += (s + 1) * (s + 2) / 2 * (smax - s + 1);
    return tot;
}

// COUNT: keep the operation counters (a separate instantiation, so the timed kernel carries none). SHARE:
// units may be shares of an item (apart, because its positions cost the others 1.5 ms of 82 in the gradient
// of an 18-atom molecule).
template <bool COUNT, bool SHARE>
__global__ void __launch_bounds__(kMmdThreads, 3) mmd_kernel(MmdArgs a)
{
    extern __shared__ double smem[];
    __shared__ int ring[kMmdRing];
    __shared__ int s_cnt[kMmdThreads / 32];
    __shared__ int4 s_unit;
    __shared__ int s_last;
    __shared__ double normA[kMmdMaxPrims], normB[kMmdMaxPrims];
    __shared__ double rcp[2 * kMmdMaxL + 1];  // 1/t
    __shared__ unsigned long long s_fl;
    constexpr int NT = kMmdThreads, NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned long long c_trip = 0, c_fl = 0;  // operation counters of this thread
    if (tid <= 2 * kMmdMaxL) rcp[tid] = 1.0 / max(tid, 1);
    for (;;) {
        if (tid == 0) {
            const int k = atomicAdd(a.queue, 1);
            s_unit = k < a.n_units ? a.units[k] : int4{-1, 0, 0, 0};
        }
        __syncthreads();
        const int4 unit = s_unit;
        if (unit.x < 0) break;
        const int share = SHARE ? unit.y & 255 : 0, nshares = SHARE ? unit.y >> 8 : 1;
        const MmdItem item = a.items[unit.x];
        const MmdClass &cl = a.classes[item.cls];
        const int la = cl.la, lb = cl.lb, S = cl.S, npairs = ncart(la) * ncart(lb);
        const int G = mmd_sum_groups(cl);
        const int *lv = a.levels + cl.lv;
        const double *Ao = a.shell_origin + 3 * item.bra;
        const double *Bo = item.ket_at_centre ? a.centre_origin + 3 * item.centre : a.shell_origin + 3 * item.ket;
        const double *Co = a.centre_origin + 3 * item.centre;
        const int npA = a.shell_nprim[item.bra], npB = a.shell_nprim[item.ket], np2 = npA * npB;
        const double *cA = a.prim_coef + a.shell_prim_off[item.bra], *xA = a.prim_alpha + a.shell_prim_off[item.bra];
        const double *cB = a.prim_coef + a.shell_prim_off[item.ket], *xB = a.prim_alpha + a.shell_prim_off[item.ket];
        const bool overlap = item.pot < 0;
        const int poff = overlap ? 0 : a.pot_prim_off[item.pot];
        const int nterms = overlap ? 1 : a.pot_nprim[item.pot], n2 = overlap ? 1 : a.pot_n2[item.pot];
        const int4 *pt = a.pairs + item.pairs;
        double *acc = smem, *ws = smem + npairs * G;
        for (int p = tid; p < npairs * G; p += NT) acc[p] = 0.0;
        if (tid < npA) normA[tid] = gaussian_norm(la, xA[tid]);
        else if (tid >= kMmdMaxPrims && tid < kMmdMaxPrims + npB) normB[tid - kMmdMaxPrims] = gaussian_norm(lb, xB[tid - kMmdMaxPrims]);
        if (COUNT && tid == 0) s_fl = 0;
        __syncthreads();
        if (COUNT) {  // operations of one triple's contraction over the item's Cartesian pairs
            unsigned long long f = 0;
            for (int p = tid; p < npairs; p += NT) {
                const int y = pt[p].y, W = (y >> 16) & 31, tx = (y >> 21) & 31, uy = (int)((unsigned)y >> 26);
                f += 3ull * (tx + 1) * (uy + 1) * (S - W + 1) + 3ull;
            }
            atomicAdd(&s_fl, f);
            __syncthreads();
        }
        // group arrays, [..][kMmdGroup]: Q-A, Q-B, Q-C, K per axis, w = c_k c_i c_j N_i N_j x
        // prefactor, 1/(2q), 2q of the 1/r^2 terms (else 0), R^n_000
        constexpr int GS = kMmdGroup;
        double *sQA = ws, *sQB = sQA + 3 * GS, *sQC = sQB + 3 * GS, *sK = sQC + 3 * GS, *sW = sK + 3 * GS, *sI = sW + GS,
               *sC = sI + GS, *sR = sC + GS, *E = sR + (S + 1) * GS;
        // candidate c of the terms from k0 on (term outer, primitive pair inner)
        auto alive = [&](int k0, int c) {
            const int k = c / np2, r = c - k * np2, i = r / npB, j = r - i * npB;
            if (!overlap && (fabs(cA[i]) < kZeroThresh || fabs(cB[j]) < kZeroThresh)) return false;
            const double al = xA[i], be = xB[j];
            const double z = overlap ? 0.0 : a.pot_alpha[poff + a.pot_perm[poff + k0 + k]];
            double ab = 0.0, ac = 0.0, bc = 0.0;
#pragma unroll
            for (int d = 0; d < 3; d++) {
                const double u = Ao[d] - Bo[d], v = Ao[d] - Co[d], w = Bo[d] - Co[d];
                ab += u * u;
                ac += v * v;
                bc += w * w;
            }
            return !(al * be * ab + al * z * ac + be * z * bc > kMmdDropArg * (al + be + z));
        };
        double *out = a.out[item.out_kind] + item.out_off;
        double *po = a.part_out + unit.z;
        // a share counts the live triples to find its parts of each kind
        int parts[2] = {0, 0};
        if (nshares > 1)
            for (int kind = 0; kind < 2; kind++) {
                const int k0 = kind == 0 ? 0 : n2, ncand = (kind == 0 ? n2 : nterms - n2) * np2;
                int n = 0;
                for (int c = tid; c - tid < ncand; c += NT) n += __syncthreads_count(c < ncand && alive(k0, c));
                const int ps = mmd_part_size((int64_t)nterms * np2, cl.lgT[kind]);
                parts[kind] = (n + ps - 1) / ps;
            }
        int part = 0;  // next part whose sums are complete
        // the sums of a part, complete after a barrier: to the output or the shares' buffer
        auto flush = [&]() {
            for (int p = tid; p < npairs; p += NT) {
                double s = 0.0;
                for (int g = 0; g < G; g++) {
                    s = g == 0 ? acc[p * G] : s + acc[p * G + g];
                    acc[p * G + g] = 0.0;
                }
                if (nshares > 1) {
                    po[part * npairs + p] = s;
                } else {
                    double *o = out + __ldg(pt + p).w;
                    *o = part == 0 ? s : *o + s;
                }
            }
            part++;
        };
        for (int kind = 0; kind < 2; kind++) {
            const int k0 = kind == 0 ? 0 : n2, ncand = (kind == 0 ? n2 : nterms - n2) * np2;
            const int lg = cl.lgT[kind], T = 1 << lg, tr = tid & (T - 1), e0 = tid >> lg, est = NT >> lg;
            const int nax = kind == 0 ? (la + 1) * (lb + 1) : mmd_e_axis(la, lb);
            double *R0 = E + cl.nE * T, *X = R0 + cl.nR0 * T, *Rb = X;  // kind 1; X shares the R levels' space
            const int ps = mmd_part_size((int64_t)nterms * np2, lg);
            // live triples lo <= index < hi of this kind: all, or a share's parts
            int lo = 0, hi = 1 << 30;
            if (nshares > 1) {
                const int k = kind == 0 ? nshares - 1 - share : share;  // who has fewer parts of one kind has more of the other
                part = parts[kind] * k / nshares;
                lo = part * ps;
                hi = parts[kind] * (k + 1) / nshares * ps;
                if (kind == 1) part += parts[0];
            }
            int head = lo, tail = lo, base = 0, seen = 0, pend = 0;
            for (;;) {
                if (tail - head < GS && base < ncand && seen < hi) {
                    // the next NT triples (term outer, primitive pair inner): keep the live ones, in order
                    const int c = base + tid;
                    bool live = false;
                    if (c < ncand) live = alive(k0, c);
                    const unsigned m = __ballot_sync(0xffffffffu, live);
                    if (lane == 0) s_cnt[warp] = __popc(m);
                    __syncthreads();
                    int pre = 0, tot = 0;
#pragma unroll
                    for (int w = 0; w < NW; w++) {
                        const int v = s_cnt[w];
                        pre += w < warp ? v : 0;
                        tot += v;
                    }
                    const int at = seen + pre + __popc(m & ((1u << lane) - 1));
                    if (live && at >= lo && at < hi) ring[at & (kMmdRing - 1)] = c;
                    seen += tot;
                    tail = max(lo, min(seen, hi));
                    base += NT;
                    __syncthreads();
                    continue;
                }
                if (tail == head) break;
                const int ng = min(GS, tail - head);
                {  // ---- scalars of the group: one thread per (triple, axis), a fourth one for the weight
                    const int t = tid & (GS - 1), d = tid / GS;
                    const bool have = t < ng;
                    const int c = ring[(head + (have ? t : 0)) & (kMmdRing - 1)];
                    const int k = c / np2, r = c - k * np2, i = r / npB, j = r - i * npB;
                    const double al = xA[i], be = xB[j];
                    const int ko = overlap ? 0 : poff + a.pot_perm[poff + k0 + k];
                    const double z = overlap ? 0.0 : a.pot_alpha[ko], q = al + be + z;
                    if (d < 3) {
                        const double A = Ao[d], B = Bo[d], C = Co[d];
                        // each product rounded, as the reference's (a A + b B + c C) / q
                        // (type1_mcmurchie_davidson.c:198); no contraction into an FMA
                        const double Q = __dadd_rn(__dadd_rn(__dmul_rn(al, A), __dmul_rn(be, B)), __dmul_rn(z, C)) / q;
                        const double ab = A - B, ac = A - C, bc = B - C;
                        const double K = exp(-((al * be) / q * ab * ab + (al * z) / q * ac * ac + (be * z) / q * bc * bc));
                        sQA[d * GS + t] = Q - A;
                        sQB[d * GS + t] = Q - B;
                        sQC[d * GS + t] = Q - C;
                        sK[d * GS + t] = K;
                    } else {
                        const double ck = overlap ? 1.0 : a.pot_coef[ko];
                        const int n = overlap ? 2 : a.pot_powers[ko];
                        const double pq = kPi / q;
                        const double pref = n == 2 ? pq * sqrt(pq) : (n == 1 ? 2.0 * pq : 2.0 * kPi15 / sqrt(q));
                        sW[t] = have ? ck * (cA[i] * cB[j]) * (normA[i] * normB[j] * pref) : 0.0;
                        sI[t] = 1.0 / (2.0 * q);
                        sC[t] = n == 0 ? 2.0 * q : 0.0;
                        sR[t] = q;
                    }
                }
                __syncthreads();
                if (COUNT && tid < ng) {
                    const int c = ring[(head + tid) & (kMmdRing - 1)], k = c / np2;
                    if (sK[tid] != 0.0 && sK[GS + tid] != 0.0 && sK[2 * GS + tid] != 0.0) {
                        const int n = overlap ? 2 : a.pot_powers[poff + a.pot_perm[poff + k0 + k]];
                        c_trip++;
                        if (overlap) c_fl += 12ull * (la + 1) * (lb + 1) + 10 + 4ull * npairs;
                        else {
                            c_fl += 40 + 5 * mmd_e_count(la, lb);
                            if (n != 2)
                                c_fl += (n == 1 ? 16ull * (S + 1) : 100ull) + 2ull * (S + 1) + 5ull * (mmd_r_size(S) - (S + 1)) + s_fl;
                            else
                                c_fl += 4ull * npairs;
                        }
                    }
                }
                if (kind == 1) {  // ---- R^n_000, n = 0..S: four threads per triple
                    const int t = tid >> 2, sub = tid & 3;
                    const double q = sR[t], dx = sQC[t], dy = sQC[GS + t], dz = sQC[2 * GS + t];
                    const bool isg = sC[t] != 0.0;
                    const double x = q * (dx * dx + dy * dy + dz * dz), q2 = isg ? 2.0 * q : -2.0 * q;
                    __syncwarp();  // q is read before sR takes the values
                    if (t < ng) {
                        if (isg) gfun_values4(x, S, sR + t, GS, sub);
                        __syncwarp(0xfu << (tid & 28));
                        for (int n = sub; n <= S; n += 4) sR[n * GS + t] = pow(q2, n) * (isg ? sR[n * GS + t] : boys(n, x));
                    }
                    __syncthreads();
                }
                for (int b0 = 0; b0 < ng; b0 += T) {
                    const int g = b0 + tr;  // this thread's triple in the group arrays
                    const bool have = g < ng;
                    for (int e = e0; e < 3; e += est) E[e * nax * T + tr] = have ? sK[e * GS + g] : 0.0;
                    if (kind == 1)
                        for (int n = e0; n <= S; n += est) {
                            const double v = have ? sR[n * GS + g] : 0.0;
                            Rb[n * T + tr] = v;
                            if (n == 0) R0[tr] = v;
                        }
                    __syncthreads();
                    const double f = sI[g];
                    if (kind == 0) {
                        const int *ol = lv + (S + 2);
                        for (int s = 1; s <= S; s++) {
                            const int n1 = ol[s + 1];
                            for (int e = ol[s] + e0; e < n1; e += est) {
                                const int2 c = __ldg(a.otab + cl.o_off + e);
                                const int ax = (c.y >> 18) & 3;
                                const double P = ((c.y >> 20) & 1 ? sQB : sQA)[ax * GS + g];
                                const double n2f = (c.y >> 10) & 15, n3f = (c.y >> 14) & 15;
                                double v = P * E[((c.x >> 10) & 1023) * T + tr];
                                v += f * (n2f * E[((c.x >> 20) & 1023) * T + tr] + n3f * E[(c.y & 1023) * T + tr]);
                                E[(c.x & 1023) * T + tr] = v;
                            }
                            __syncthreads();
                        }
                    } else {
                        // ---- step s: E wavefront i + j = s and R level s
                        const int *rl = lv + 2 * (S + 2);
                        const double c2q = sC[g];
                        const bool isg = c2q != 0.0;
                        for (int s = 1; s <= S; s++) {
                            const int n1 = lv[s + 1];
                            for (int e = lv[s] + e0; e < n1; e += est) {
                                const int2 c = __ldg(a.etab + cl.e_off + e);
                                const int ax = (c.y >> 13) & 3, src = (c.x >> 13) & 8191;
                                double v;
                                if (c.x & (1 << 30)) {
                                    v = ((c.y >> 20) & 1 ? sQB : sQA)[ax * GS + g] * E[src * T + tr];
                                    if ((c.y >> 24) & 1) v += E[(src + 1) * T + tr];
                                } else {
                                    const double ii = (c.y >> 20) & 15, jj = (c.y >> 24) & 15;
                                    v = f * rcp[(c.y >> 15) & 31] * (ii * E[src * T + tr] + jj * E[(c.y & 8191) * T + tr]);
                                }
                                E[(c.x & 8191) * T + tr] = v;
                            }
                            double *dst = Rb + (s % 3) * cl.maxlev * T;
                            const double *p1 = Rb + ((s + 2) % 3) * cl.maxlev * T, *p2 = Rb + ((s + 1) % 3) * cl.maxlev * T;
                            const int m0 = rl[s], m1 = rl[s + 1], ne1 = s * (s + 1) / 2, ne2 = (s - 1) * s / 2;
                            for (int e = m0 + e0; e < m1; e += est) {
                                const int2 c = __ldg(a.rtab + cl.r_off + e);
                                const int k = (c.y >> 14) & 31, r0d = c.y & 8191, s1 = c.x & 0xffff, s2 = (int)((unsigned)c.x >> 16);
                                double v = 0.0;
                                if (k > 1) {
                                    double d2 = p2[(s2 + ne2) * T + tr];
                                    if (isg) d2 = __fma_rn(-c2q, p2[s2 * T + tr], d2);
                                    v = (k - 1) * d2;
                                }
                                double d1 = p1[(s1 + ne1) * T + tr];
                                if (isg) d1 = __fma_rn(-c2q, p1[s1 * T + tr], d1);
                                v = __fma_rn(sQC[((c.y >> 19) & 3) * GS + g], d1, v);
                                dst[(e - m0) * T + tr] = v;
                                if (r0d != kMmdNoR0) R0[r0d * T + tr] = v;
                            }
                            __syncthreads();
                        }
                        // ---- X[(az, bz)][t][u] = sum_v E^z_v R^0_tuv (the R levels are consumed)
                        for (int e = e0; e < cl.nX; e += est) {
                            const int2 c = __ldg(a.ztab + cl.z_off + e);
                            const double *r = R0 + (c.x & 0xffff) * T + tr, *z = E + ((unsigned)c.x >> 16) * T + tr;
                            double v = z[0] * r[0];
                            for (int u = 1; u <= c.y; u++) v += z[u * T] * r[u * T];
                            X[e * T + tr] = v;
                        }
                        __syncthreads();
                    }
                    // ---- Cartesian pairs: one thread per (pair, triple); the batch's triples are added by a
                    // shuffle tree, then to the pair's running sum
                    const double w = sW[g];
                    const int rounds = (npairs * T + NT - 1) / NT;
                    for (int rd = 0, p = e0; rd < rounds; rd++, p += est) {
                        double s = 0.0;
                        if (p < npairs) {
                            const int4 d = __ldg(pt + p);
                            if (kind == 0) {
                                s = E[(d.z & 1023) * T + tr] * E[((d.z >> 10) & 1023) * T + tr] * E[((d.z >> 20) & 1023) * T + tr];
                            } else {
                                const double *ex = E + (d.x & 0xffff) * T + tr, *ey = E + ((unsigned)d.x >> 16) * T + tr;
                                const double *x = X + (d.y & 0xffff) * T + tr;
                                const int W = (d.y >> 16) & 31, tx = (d.y >> 21) & 31, uy = (int)((unsigned)d.y >> 26);
                                for (int t = 0; t <= tx; t++) {
                                    double sy = ey[0] * x[0];
                                    for (int u = 1; u <= uy; u++) sy += ey[u * T] * x[u * T];
                                    s += ex[t * T] * sy;
                                    x += (W + 1 - t) * T;
                                }
                            }
                            s *= w;
                        }
                        for (int o = min(T, 32) >> 1; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
                        if (p < npairs && (tr & 31) == 0) acc[p * G + (tr >> 5)] += s;
                    }
                    __syncthreads();  // the batch's tables are consumed
                    pend += T;
                    if (pend == ps) {
                        flush();
                        pend = 0;
                    }
                }
                head += ng;
            }
            if (pend > 0) flush();
        }
        if (part == 0 && nshares == 1)  // no triple is left
            for (int p = tid; p < npairs; p += NT) out[__ldg(pt + p).w] = 0.0;
        if (nshares > 1) {  // the share that comes last adds all parts, in order
            __threadfence();
            __syncthreads();
            if (tid == 0) s_last = atomicAdd(a.part_cnt + unit.w, 1) == nshares - 1;
            __syncthreads();
            if (s_last) {
                __threadfence();
                const int np_all = parts[0] + parts[1];
                for (int p = tid; p < npairs; p += NT) {
                    double s = 0.0;
                    for (int q = 0; q < np_all; q++) s = q == 0 ? __ldcg(po + p) : s + __ldcg(po + q * npairs + p);
                    out[__ldg(pt + p).w] = s;
                }
            }
        }
        __syncthreads();  // acc and s_unit are consumed
    }
    if (COUNT && a.counters) {
        for (int o = 16; o > 0; o >>= 1) {
            c_trip += __shfl_down_sync(0xffffffffu, c_trip, o);
            c_fl += __shfl_down_sync(0xffffffffu, c_fl, o);
        }
        if (lane == 0) {
            atomicAdd(a.counters + kRadCntMmdTriples, c_trip);
            atomicAdd(a.counters + kRadCntMmdFlops, c_fl);
        }
    }
}

}  // namespace grpp

// One-electron integrals over contracted Cartesian Gaussian shell pairs (FP64).
//
//   onee_os_kernel     overlap, kinetic energy and momentum blocks by the Obara-Saika
//                      recurrences (libgrpp/overlap.c:39-139, kinetic.c:48-162,
//                      momentum.c:48-181). One warp per shell pair: up to ten primitive pairs
//                      at a time, one lane per pair and axis builds the tables S_ij (and D1_ij
//                      or D2_ij) in shared memory, then every lane owns Cartesian pairs of
//                      the block and adds c_i c_j N_i N_j S S S with libgrpp's rounding
//                      (primitive pairs in order, products left to right, no fused multiply-add).
//   type1_ang_kernel   k-independent angular factors of the numeric type 1 integral,
//                      A1[lambda][mu][IJK] = sum_rst y_{lambda mu, rst} I(I+r, J+s, K+t)
//                      (libgrpp/angular_integrals.c:35-56), once per batch.
//   numeric type 1 integrals <A| V(|r - C|) |B> of a radially local potential: a GRPP's U_L, or
//                      the electrostatic potential of a point, charged-ball, Gaussian, Fermi or
//                      Fermi-bubble nucleus (libgrpp/nuclear_models.c), by libgrpp's
//                      per-primitive-pair scheme (type1_integrals.c:144-270,
//                      radial_type1_integral.c:73-325): radial integrals Q(lambda, N) of the
//                      pair on the nested Log3 grid (2047 -> 4095 -> 8191 points, stop at
//                      |S_L - S_{L-1}| <= tol), then the binomial re-centring of both shells on
//                      C with the angular factors of k = -2 (a CA + b CB). Five kernels:
//   t1_points_kernel   r and r^N of the 8191 grid points, once per call
//   t1_wpot_kernel     weight x potential at every point, once per centre
//   t1_radial_kernel   Q(lambda, N): one warp per primitive pair, every sum in point order
//   t1_assemble_kernel re-centring: one block per four primitive pairs of a task
//   t1_sum_kernel      the pairs' contributions added in libgrpp's order
#pragma once

#include "angular.cuh"
#include "nucmodel.h"

namespace grpp {

__device__ __forceinline__ double rn_add(double x, double y) { return __dadd_rn(x, y); }
__device__ __forceinline__ double rn_mul(double x, double y) { return __dmul_rn(x, y); }

// ------------------------------------------------------------------ Obara-Saika
enum OneeKind : int { kOneeOverlap = 0, kOneeKinetic = 1, kOneeMomentum = 2 };

struct OneeArgs {
    int n_tasks, kind;
    const int *task_a, *task_b;
    const int64_t *out_off;
    const int *shell_L, *shell_nprim, *shell_prim_off, *shell_cart_off;
    const double *prim_coef, *prim_alpha, *shell_origin;
    const int8_t *cart;
    double *out0, *out1, *out2;
};

constexpr int kOneeWarps = 4;
constexpr int kOneeTab = 1350;  // doubles of tables per warp
constexpr int kOneeQ = 10;      // primitive pairs at a time: three lanes each
static_assert(3 * (((kMaxL + 3) * (kMaxL + 3) + (kMaxL + 1) * (kMaxL + 1)) | 1) <= kOneeTab, "tables of one primitive pair");

// Bound by the chain of the recurrences and by issue of the component products, about evenly
// at six or more primitive pairs. Before, three lanes built one primitive pair's tables while 29 waited, every
// lane computed the norms, and each product was added to the block in global memory: every
// ordered shell pair of 48 atoms (s..g) took 3.07 ms, 0.54 ms here. 1350 doubles hold six pairs of g
// shells and leave room for five blocks on an SM.
__global__ void __launch_bounds__(32 * kOneeWarps) onee_os_kernel(OneeArgs a)
{
    __shared__ double s_tab[kOneeWarps][kOneeTab];
    __shared__ double s_fac[kOneeWarps][2 * kOneeQ];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ext = a.kind == kOneeKinetic ? 2 : (a.kind == kOneeMomentum ? 1 : 0);
    double *tab = s_tab[w], *fac = s_fac[w];
    for (int t = blockIdx.x * kOneeWarps + w; t < a.n_tasks; t += gridDim.x * kOneeWarps) {
        const int A = a.task_a[t], B = a.task_b[t];
        const int la = a.shell_L[A], lb = a.shell_L[B], nB = ncart(lb), np = ncart(la) * nB;
        const double *oA = a.shell_origin + 3 * A, *oB = a.shell_origin + 3 * B;
        const int8_t *ca = a.cart + 3 * a.shell_cart_off[A], *cb = a.cart + 3 * a.shell_cart_off[B];
        double *o0 = a.out0 + a.out_off[t];
        double *o1 = a.kind == kOneeMomentum ? a.out1 + a.out_off[t] : nullptr;
        double *o2 = a.kind == kOneeMomentum ? a.out2 + a.out_off[t] : nullptr;
        const int pa = a.shell_prim_off[A], pb = a.shell_prim_off[B], nb = a.shell_nprim[B], npr = a.shell_nprim[A] * nb;
        // per pair and axis: S[ii][jj], rows of ws, then D[ii][jj], rows of wd
        const int ws = lb + ext + 1, wd = lb + 1, nS = (la + ext + 1) * ws, axis = (nS + (la + 1) * wd) | 1;
        const int nq = min(kOneeQ, kOneeTab / (3 * axis));
        if (npr == 0)
            for (int p = lane; p < np; p += 32) {
                o0[p] = 0.0;
                if (o1) {
                    o1[p] = 0.0;
                    o2[p] = 0.0;
                }
            }
        for (int q0 = 0; q0 < npr; q0 += nq) {
            const int cnt = min(nq, npr - q0);
            __syncwarp();
            if (lane < 3 * cnt) {
                const int q = lane / 3, c = lane - 3 * q, i = (q0 + q) / nb, j = q0 + q - i * nb;
                double *S = tab + lane * axis, *D = S + nS;
                const double ai = a.prim_alpha[pa + i], aj = a.prim_alpha[pb + j];
                const double p = ai + aj, mu = ai * aj / p;
                const double P = rn_add(rn_mul(ai, oA[c]), rn_mul(aj, oB[c])) / p;
                const double xab = oA[c] - oB[c], xpa = P - oA[c], xpb = P - oB[c], pf = 1.0 / (2.0 * p);
                double s1 = sqrt(kPi / p) * exp(-mu * xab * xab), s2 = 0.0;
                S[0] = s1;
                for (int jj = 1; jj < ws; jj++) {
                    double s = rn_mul(xpb, s1);
                    if (jj > 1) s = rn_add(s, rn_mul(rn_mul(jj - 1, pf), s2));
                    S[jj] = s;
                    s2 = s1;
                    s1 = s;
                }
                for (int ii = 1; ii <= la + ext; ii++) {
                    const double fi = rn_mul(ii - 1, pf);
                    double *r = S + ii * ws;
#pragma unroll 4
                    for (int jj = 0; jj < ws; jj++) {
                        double s = rn_mul(xpa, r[jj - ws]);
                        if (ii > 1) s = rn_add(s, rn_mul(fi, r[jj - 2 * ws]));
                        if (jj > 0) s = rn_add(s, rn_mul(rn_mul(jj, pf), r[jj - ws - 1]));
                        r[jj] = s;
                    }
                }
                if (a.kind == kOneeKinetic) {
                    for (int ii = 0; ii <= la; ii++)
                        for (int jj = 0; jj <= lb; jj++) {
                            double d = rn_mul(rn_mul(4.0 * ai, ai), S[(ii + 2) * ws + jj]);
                            d = rn_add(d, -rn_mul(rn_mul(2.0 * ai, 2 * ii + 1), S[ii * ws + jj]));
                            if (ii >= 2) d = rn_add(d, rn_mul(ii * (ii - 1), S[(ii - 2) * ws + jj]));
                            D[ii * wd + jj] = d;
                        }
                } else if (a.kind == kOneeMomentum) {
                    for (int ii = 0; ii <= la; ii++)
                        for (int jj = 0; jj <= lb; jj++) {
                            double d = rn_mul(2.0 * ai, S[(ii + 1) * ws + jj]);
                            if (ii >= 1) d = rn_add(d, -rn_mul(ii, S[(ii - 1) * ws + jj]));
                            D[ii * wd + jj] = d;
                        }
                }
            }
            if (lane < cnt) {
                const int i = (q0 + lane) / nb, j = q0 + lane - i * nb;
                const double NA = gaussian_norm(la, a.prim_alpha[pa + i]), NB = gaussian_norm(lb, a.prim_alpha[pb + j]);
                fac[2 * lane] = rn_mul(a.prim_coef[pa + i], a.prim_coef[pb + j]);
                fac[2 * lane + 1] = a.kind == kOneeOverlap ? rn_mul(NA, NB)
                                                           : rn_mul(a.kind == kOneeKinetic ? -0.5 * NA : -NA, NB);
            }
            __syncwarp();
            for (int p = lane; p < np; p += 32) {
                const int m = p / nB, n = p - m * nB;
                const int x1 = ca[3 * m], y1 = ca[3 * m + 1], z1 = ca[3 * m + 2];
                const int x2 = cb[3 * n], y2 = cb[3 * n + 1], z2 = cb[3 * n + 2];
                const double *Sx = tab + x1 * ws + x2, *Sy = tab + axis + y1 * ws + y2, *Sz = tab + 2 * axis + z1 * ws + z2;
                const double *Dx = tab + nS + x1 * wd + x2, *Dy = tab + axis + nS + y1 * wd + y2,
                             *Dz = tab + 2 * axis + nS + z1 * wd + z2;
                double v0 = 0.0, v1 = 0.0, v2 = 0.0;
                if (q0 > 0) {
                    v0 = o0[p];
                    if (o1) {
                        v1 = o1[p];
                        v2 = o2[p];
                    }
                }
                for (int q = 0; q < cnt; q++) {
                    const int o = 3 * q * axis;
                    const double cc = fac[2 * q], f = fac[2 * q + 1], sx = Sx[o], sy = Sy[o], sz = Sz[o];
                    if (a.kind == kOneeOverlap) {
                        v0 = rn_add(v0, rn_mul(cc, rn_mul(rn_mul(rn_mul(f, sx), sy), sz)));
                    } else if (a.kind == kOneeKinetic) {
                        double s = rn_mul(rn_mul(Dx[o], sy), sz);
                        s = rn_add(s, rn_mul(rn_mul(sx, Dy[o]), sz));
                        s = rn_add(s, rn_mul(rn_mul(sx, sy), Dz[o]));
                        v0 = rn_add(v0, rn_mul(cc, rn_mul(f, s)));
                    } else {
                        v0 = rn_add(v0, rn_mul(cc, rn_mul(rn_mul(rn_mul(f, Dx[o]), sy), sz)));
                        v1 = rn_add(v1, rn_mul(cc, rn_mul(rn_mul(rn_mul(f, sx), Dy[o]), sz)));
                        v2 = rn_add(v2, rn_mul(cc, rn_mul(rn_mul(rn_mul(f, sx), sy), Dz[o])));
                    }
                }
                o0[p] = v0;
                if (o1) {
                    o1[p] = v1;
                    o2[p] = v2;
                }
            }
        }
    }
}

// ------------------------------------------------------------------ numeric type 1
constexpr int kT1MaxLam = 12;       // L_A + L_B <= 12
constexpr int kT1Pts = 8192;        // row length of the point tables (8191 points in order of evaluation)
constexpr int kT1Warps = 4;         // warps of a radial block
constexpr int kT1Group = 4;         // primitive pairs of an assembly block
constexpr int kT1AsmThreads = 128;
constexpr int kT1PowRow = kMaxL + 1;  // powers 0..kMaxL of one component of CA or CB: one shell may have all of L_A + L_B

struct Type1NumArgs {
    int n_tasks, model;
    const int *task_a, *task_b, *task_c;
    const int64_t *out_off;
    const int *shell_L, *shell_nprim, *shell_prim_off, *shell_cart_off;
    const double *prim_coef, *prim_alpha, *shell_origin;
    const int8_t *cart;
    const double *centre_origin;
    const double *centre_param;        // [n_centres][4]: Z and the model's parameters
    const int *centre_pot_off, *centre_pot_n;  // kPotGrpp: the centre's U_L terms
    const int *pot_pow;
    const double *pot_coef, *pot_alpha;
    const double *fermi;               // [kFermiNX][kFermiNK]
    const double *ang1;                // type1_ang_kernel output for lmax_tab
    int lmax_tab;
    double tol;                        // radial stop tolerance (libgrpp_params.radial_tolerance)
    double pair_skip;                  // primitive pairs with |c_i c_j| below it are skipped
    // one chunk of tasks (the task arrays above and these start at it)
    const int64_t *unit_off, *group_off;  // [n_tasks + 1] first primitive pair / assembly block of a task
    const int64_t *scr_off;               // per task: doubles into scratch, [pair][nq + block size]
    const int *slot;                      // per task: row of wpot
    const int *slot_centre;
    int n_slots;
    double *points;                       // r, then r^0 .. r^lmax_tab: rows of kT1Pts
    double *wpot;                         // [n_slots][kT1Pts]
    double *scratch;
    double *out;
};

// Q(lambda, N) entries that the angular factors read: lambda of N's parity (for the others every
// integral over the sphere has an odd power and vanishes)
__host__ __device__ inline int t1_row(int lmax) { return lmax / 2 + 1; }
__host__ __device__ inline int t1_nq(int lmax) { return (lmax + 1) * t1_row(lmax); }

// the task of item u, off[t] <= u < off[t + 1] counted from off[0]
__device__ __forceinline__ int t1_find(const int64_t *off, int n, int64_t u)
{
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int m = (lo + hi) / 2;
        if (off[m] - off[0] <= u) lo = m;
        else hi = m;
    }
    return lo;
}

// A1 layout for lmax_tab = Lt: [lambda (0..Lt)][mu (0..2 Lt)][IJK index among I+J+K <= Lt]
__host__ __device__ inline int64_t ang1_index(int Lt, int lam, int mu_off, int ijk)
{
    return ((int64_t)lam * (2 * Lt + 1) + mu_off) * n_abc(Lt) + ijk;
}

__global__ void type1_ang_kernel(int Lt, double *A1)
{
    const int64_t n = (int64_t)(Lt + 1) * (2 * Lt + 1) * n_abc(Lt);
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
        const int ijk = (int)(e % n_abc(Lt));
        const int mu_off = (int)((e / n_abc(Lt)) % (2 * Lt + 1));
        const int lam = (int)(e / ((int64_t)n_abc(Lt) * (2 * Lt + 1)));
        const int mu = mu_off - lam;
        double v = 0.0;
        if (mu <= lam) {
            // (I, J, K) of index ijk: lexicographic among I+J+K <= Lt
            int I = 0, J = 0, K = 0, q = 0;
            for (int a = 0; a <= Lt && q <= ijk; a++)
                for (int b = 0; a + b <= Lt && q <= ijk; b++)
                    for (int c = 0; a + b + c <= Lt && q <= ijk; c++, q++)
                        if (q == ijk) {
                            I = a;
                            J = b;
                            K = c;
                        }
            const int nc = ncart(lam);
            const int8_t *cc = c_tab.rsh_comb + 3 * c_tab.rsh_comb_off[lam];
            const double *y = c_tab.rsh_coef + c_tab.rsh_off[lam] + (mu + lam) * nc;
            for (int r = 0; r < nc; r++) v = rn_add(v, rn_mul(y[r], usp_integral(I + cc[3 * r], J + cc[3 * r + 1], K + cc[3 * r + 2])));
        }
        A1[e] = v;
    }
}

// grid points of the three levels in order of evaluation: 2047, then 2048 and 4096 new ones
__device__ __forceinline__ void t1_point(int q, double &r, double &w)
{
    const int nr = q < 2047 ? 2047 : (q < 4095 ? 4095 : 8191);
    const int ip = q < 2047 ? q + 1 : (q < 4095 ? 2 * (q - 2047) + 1 : 2 * (q - 4095) + 1);
    const double xi = ip / (nr + 1.0), xi3 = xi * xi * xi, ln = log(1 - xi3);
    const double R = 5.0, R3 = R * R * R;
    w = 3 * R3 * xi * xi * ln * ln / ((1 - xi3) * (nr + 1.0));
    r = -R * ln;
}

__global__ void t1_points_kernel(Type1NumArgs a)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= kT1Pts - 1) return;
    double r, w;
    t1_point(q, r, w);
    a.points[q] = r;
    for (int n = 0; n <= a.lmax_tab; n++) a.points[(int64_t)(1 + n) * kT1Pts + q] = pow(r, (double)n);
}

__global__ void t1_wpot_kernel(Type1NumArgs a)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= kT1Pts - 1) return;
    double r, w;
    t1_point(q, r, w);
    for (int s = blockIdx.y; s < a.n_slots; s += gridDim.y) {
        const int C = a.slot_centre[s];
        double pot;
        if (a.model == kPotGrpp) {
            pot = 0.0;
            const int o = a.centre_pot_off[C];
            const double r2 = r * r;
            for (int u = 0; u < a.centre_pot_n[C]; u++)
                pot = rn_add(pot, rn_mul(rn_mul(a.pot_coef[o + u], pow(r, (double)(a.pot_pow[o + u] - 2))),
                                         exp(-a.pot_alpha[o + u] * r2)));
        } else {
            pot = nuclear_potential(a.model, a.centre_param + 4 * C, r, a.fermi);
        }
        a.wpot[(int64_t)s * kT1Pts + q] = w * pot;
    }
}

// geometry of one primitive pair, as every kernel below forms it
struct T1Pair {
    double CA[3], CB[3], CA2, CB2, kv[3], k, ai, aj, ci, cj;
    bool skip;
};

__device__ __forceinline__ T1Pair t1_pair(const Type1NumArgs &a, int A, int B, int C, int j)
{
    T1Pair p;
    const double *oA = a.shell_origin + 3 * A, *oB = a.shell_origin + 3 * B, *oC = a.centre_origin + 3 * C;
    const double CAx = oC[0] - oA[0], CAy = oC[1] - oA[1], CAz = oC[2] - oA[2];
    const double CBx = oC[0] - oB[0], CBy = oC[1] - oB[1], CBz = oC[2] - oB[2];
    p.CA2 = CAx * CAx + CAy * CAy + CAz * CAz;
    p.CB2 = CBx * CBx + CBy * CBy + CBz * CBz;
    const int nb = a.shell_nprim[B], i = j / nb, pa = a.shell_prim_off[A] + i, pb = a.shell_prim_off[B] + j - i * nb;
    p.ci = a.prim_coef[pa];
    p.cj = a.prim_coef[pb];
    p.ai = a.prim_alpha[pa];
    p.aj = a.prim_alpha[pb];
    p.skip = fabs(p.ci * p.cj) < a.pair_skip;
    const double kv[3] = {-2.0 * fma(p.ai, CAx, rn_mul(p.aj, CBx)), -2.0 * fma(p.ai, CAy, rn_mul(p.aj, CBy)),
                          -2.0 * fma(p.ai, CAz, rn_mul(p.aj, CBz))};
    p.k = sqrt(kv[0] * kv[0] + kv[1] * kv[1] + kv[2] * kv[2]);
    const double ca[3] = {CAx, CAy, CAz}, cb[3] = {CBx, CBy, CBz};
    for (int d = 0; d < 3; d++) {
        p.CA[d] = ca[d];
        p.CB[d] = cb[d];
        p.kv[d] = kv[d];
    }
    return p;
}

// Radial integrals, one warp per primitive pair: the lanes evaluate 32 points, then each lane adds
// the 32 terms of its entries in point order, so every sum has libgrpp's order. Bound by the FP64
// pipe (Bessel rows and the 2 operations per entry and point); the chain of additions of one pair
// hides behind the other warps of the SM. A batch whose integrand underflows everywhere adds
// zeros and is passed over. Before, a block walked all pairs of a task one after another with
// one thread per entry, and evaluated the potential and the powers of r for every pair: 300 tasks
// of s..f shells with 36 pairs each took 33.7 ms; 3.26 ms here and 0.13 ms in the kernels around it.
// The kernels keep the operations of one pair's sums and factors as they were (k = -2 (a CA + b CB) with one
// rounding of b CB included): re-centring amplifies their last bits by up to 1e7.
template <int E>
__global__ void __launch_bounds__(32 * kT1Warps) t1_radial_kernel(Type1NumArgs a, int64_t n_units)
{
    extern __shared__ double t1_sm[];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int64_t u = (int64_t)blockIdx.x * kT1Warps + wp;
    if (u >= n_units) return;
    const int t = t1_find(a.unit_off, a.n_tasks, u), j = (int)(u - (a.unit_off[t] - a.unit_off[0]));
    const int A = a.task_a[t], B = a.task_b[t];
    const int la = a.shell_L[A], lb = a.shell_L[B], lmax = la + lb, nq = t1_nq(lmax);
    const T1Pair p = t1_pair(a, A, B, a.task_c[t], j);
    if (p.skip) return;
    const double Dabc = 4 * kPi * gaussian_norm(la, p.ai) * gaussian_norm(lb, p.aj);
    double *wr = t1_sm + wp * 2 * (a.lmax_tab + 1) * 33, *bes = wr + (lmax + 1) * 33;
    const double *wpot = a.wpot + (int64_t)a.slot[t] * kT1Pts, *rp = a.points + kT1Pts;
    double sum[E], prev[E];
    bool act[E];
    int rw[E], rb[E];
#pragma unroll
    for (int x = 0; x < E; x++) {
        const int e = lane + 32 * x;
        const int N = e / t1_row(lmax), lam = (N & 1) + 2 * (e - N * t1_row(lmax));
        sum[x] = prev[x] = 0.0;
        act[x] = e < nq && lam <= lmax;
        rw[x] = act[x] ? N * 33 : 0;
        rb[x] = act[x] ? lam * 33 : 0;
    }
    int base = 0;
    for (int level = 0; level < 3; level++) {
        const int npts = level == 0 ? 2047 : (level == 1 ? 2048 : 4096);
        if (level > 0) {
#pragma unroll
            for (int x = 0; x < E; x++)
                if (act[x]) {
                    prev[x] = sum[x];
                    sum[x] = 0.5 * sum[x];
                }
        }
        for (int c0 = 0; c0 < npts; c0 += 32) {
            const int q = base + c0 + lane;
            const bool in = c0 + lane < npts;
            double r = 1.0, wpg = 0.0;
            if (in) {
                r = a.points[q];
                const double power = rn_add(rn_add(rn_add(rn_mul(p.k, r), -rn_mul(rn_mul(p.ai + p.aj, r), r)), -rn_mul(p.ai, p.CA2)),
                                            -rn_mul(p.aj, p.CB2));
                const double gto = Dabc * exp(power);
                wpg = wpot[q] * gto;
            }
            if (!__any_sync(0xffffffffu, wpg != 0.0)) continue;
            if (in) {
                double M[kT1MaxLam + 1];
                bessel_scaled_row<kT1MaxLam>(lmax, r * p.k, M);
#pragma unroll
                for (int l = 0; l <= kT1MaxLam; l++)
                    if (l <= lmax) {
                        bes[l * 33 + lane] = M[l];
                        wr[l * 33 + lane] = rn_mul(wpg, rp[(int64_t)l * kT1Pts + q]);
                    }
            }
            __syncwarp();
            const int cn = min(32, npts - c0);
            if (cn == 32) {
#pragma unroll 8
                for (int i = 0; i < 32; i++)
#pragma unroll
                    for (int x = 0; x < E; x++) {
                        const double v = rn_add(sum[x], rn_mul(wr[rw[x] + i], bes[rb[x] + i]));
                        if (act[x]) sum[x] = v;
                    }
            } else {
                for (int i = 0; i < cn; i++)
#pragma unroll
                    for (int x = 0; x < E; x++) {
                        const double v = rn_add(sum[x], rn_mul(wr[rw[x] + i], bes[rb[x] + i]));
                        if (act[x]) sum[x] = v;
                    }
            }
            __syncwarp();
        }
        base += npts;
        if (level > 0) {
            bool any = false;
#pragma unroll
            for (int x = 0; x < E; x++) {
                if (act[x] && fabs(sum[x] - prev[x]) <= a.tol) act[x] = false;
                any |= act[x];
            }
            if (!__any_sync(0xffffffffu, any)) break;
        }
    }
    double *Q = a.scratch + a.scr_off[t] + (int64_t)j * (nq + ncart(la) * ncart(lb));
#pragma unroll
    for (int x = 0; x < E; x++)
        if (lane + 32 * x < nq) Q[lane + 32 * x] = sum[x];
}

__host__ __device__ inline int t1_radial_smem(int lmax) { return kT1Warps * 2 * (lmax + 1) * 33; }
__host__ __device__ inline int t1_assemble_smem(int lmax)
{
    return 6 * kT1PowRow + kT1Group * (3 * (lmax + 1) + (lmax + 1) * (lmax + 1) + n_abc(lmax)) + (n_abc(lmax) + 1) / 2;
}

// Binomial re-centring of both shells on C (type1_integrals.c:206-262). The inner sum over lambda
// depends on (I, J, K) only, so it is tabulated per primitive pair before the components are
// visited, and the binomial factors of a component are formed once for the block's four pairs.
__global__ void __launch_bounds__(kT1AsmThreads) t1_assemble_kernel(Type1NumArgs a, int64_t n_groups)
{
    extern __shared__ double t1_sm[];
    const int tid = threadIdx.x;
    for (int64_t gi = blockIdx.x; gi < n_groups; gi += gridDim.x) {
        const int t = t1_find(a.group_off, a.n_tasks, gi), j0 = (int)(gi - (a.group_off[t] - a.group_off[0])) * kT1Group;
        const int A = a.task_a[t], B = a.task_b[t], C = a.task_c[t];
        const int la = a.shell_L[A], lb = a.shell_L[B], nA = ncart(la), nB = ncart(lb), np = nA * nB;
        const int lmax = la + lb, nq = t1_nq(lmax), nijk = n_abc(lmax), nlm = (lmax + 1) * (lmax + 1);
        const int nj = min(kT1Group, (int)(a.unit_off[t + 1] - a.unit_off[t]) - j0);
        double *pw = t1_sm, *up = pw + 6 * kT1PowRow, *rsh = up + kT1Group * 3 * (lmax + 1), *sq = rsh + kT1Group * nlm;
        int *tij = (int *)(sq + kT1Group * nijk);  // index under lmax_tab, degree in the top byte
        double *scr = a.scratch + a.scr_off[t] + (int64_t)j0 * (nq + np);
        __syncthreads();
        if (tid < 6) {
            const T1Pair p = t1_pair(a, A, B, C, j0);
            const double u = tid < 3 ? p.CA[tid] : p.CB[tid - 3];
            for (int n = 0; n <= (tid < 3 ? la : lb); n++) pw[tid * kT1PowRow + n] = pow(u, (double)n);
        } else if (tid >= 32 && tid < 32 + 3 * nj) {
            // powers of the unit vector k/|k| (spherical_harmonics.c:172-220)
            const int c = (tid - 32) / 3, d = (tid - 32) % 3;
            const T1Pair p = t1_pair(a, A, B, C, j0 + c);
            const double ux = p.k > kZeroThresh ? p.kv[d] / p.k : 0.0;
            double v = 1.0;
            for (int n = 0; n <= lmax; n++) {
                up[(c * 3 + d) * (lmax + 1) + n] = v;
                v *= ux;
            }
        }
        for (int I = tid; I < (lmax + 1) * (lmax + 1); I += kT1AsmThreads) {
            const int x = I / (lmax + 1), y = I - x * (lmax + 1);
            for (int z = 0; x + y + z <= lmax; z++)
                tij[abc_index(lmax, x, y, z)] = abc_index(a.lmax_tab, x, y, z) | (x + y + z) << 24;
        }
        __syncthreads();
        for (int e = tid; e < nlm * nj; e += kT1AsmThreads) {
            const int c = e / nlm, lm = e - c * nlm;
            int l = (int)sqrtf((float)lm);
            while (l * l > lm) l--;
            while ((l + 1) * (l + 1) <= lm) l++;
            const int mu = lm - l * l - l, nc = ncart(l);
            const int8_t *cc = c_tab.rsh_comb + 3 * c_tab.rsh_comb_off[l];
            const double *y = c_tab.rsh_coef + c_tab.rsh_off[l] + (mu + l) * nc;
            const double *u = up + c * 3 * (lmax + 1);
            double v = 0.0;
            for (int q = 0; q < nc; q++)
                v = rn_add(v, rn_mul(rn_mul(rn_mul(y[q], u[cc[3 * q]]), u[lmax + 1 + cc[3 * q + 1]]), u[2 * (lmax + 1) + cc[3 * q + 2]]));
            rsh[e] = v;
        }
        __syncthreads();
        for (int e = tid; e < nijk; e += kT1AsmThreads) {
            const int ti = tij[e] & 0xffffff, N = tij[e] >> 24;
            double s[kT1Group];
            for (int c = 0; c < kT1Group; c++) s[c] = 0.0;
            for (int l = N & 1; l <= lmax; l += 2) {
                double om[kT1Group];
#pragma unroll
                for (int c = 0; c < kT1Group; c++) om[c] = 0.0;
                for (int m = 0; m <= 2 * l; m++) {
                    const double f = a.ang1[ang1_index(a.lmax_tab, l, m, ti)];
                    if (f == 0.0) continue;
#pragma unroll
                    for (int c = 0; c < kT1Group; c++)
                        if (c < nj) om[c] = rn_add(om[c], rn_mul(f, rsh[c * nlm + l * l + m]));
                }
#pragma unroll
                for (int c = 0; c < kT1Group; c++)
                    if (c < nj) {
                        const double Q = scr[(int64_t)c * (nq + np) + N * t1_row(lmax) + l / 2];
                        if (!(fabs(Q) < 1e-16)) s[c] = rn_add(s[c], rn_mul(om[c], Q));
                    }
            }
#pragma unroll
            for (int c = 0; c < kT1Group; c++) sq[c * nijk + e] = s[c];
        }
        __syncthreads();
        double cc[kT1Group];
        bool skip[kT1Group];
#pragma unroll
        for (int c = 0; c < kT1Group; c++) {
            const T1Pair p = t1_pair(a, A, B, C, j0 + min(c, nj - 1));
            cc[c] = p.ci * p.cj;
            skip[c] = p.skip;
        }
        const int8_t *ca = a.cart + 3 * a.shell_cart_off[A], *cb = a.cart + 3 * a.shell_cart_off[B];
        for (int p = tid; p < np; p += kT1AsmThreads) {
            const int m = p / nB, n = p - m * nB;
            const int nxA = ca[3 * m], nyA = ca[3 * m + 1], nzA = ca[3 * m + 2];
            const int nxB = cb[3 * n], nyB = cb[3 * n + 1], nzB = cb[3 * n + 2];
            double chi[kT1Group];
#pragma unroll
            for (int c = 0; c < kT1Group; c++) chi[c] = 0.0;
            for (int aa = 0; aa <= nxA; aa++) {
                const double C1 = c_tab.binom[nxA * kBinN + aa], P1 = pw[nxA - aa];
                for (int bb = 0; bb <= nyA; bb++) {
                    const double C2 = C1 * c_tab.binom[nyA * kBinN + bb], P2 = pw[kT1PowRow + nyA - bb];
                    for (int cq = 0; cq <= nzA; cq++) {
                        const double C3 = C2 * c_tab.binom[nzA * kBinN + cq], P3 = pw[2 * kT1PowRow + nzA - cq];
                        for (int d = 0; d <= nxB; d++) {
                            const double C4 = C3 * c_tab.binom[nxB * kBinN + d], P4 = pw[3 * kT1PowRow + nxB - d];
                            for (int e = 0; e <= nyB; e++) {
                                const double C5 = C4 * c_tab.binom[nyB * kBinN + e], P5 = pw[4 * kT1PowRow + nyB - e];
                                const double *row = sq + abc_index(lmax, aa + d, bb + e, cq);
                                for (int f = 0; f <= nzB; f++) {
                                    const double C6 = c_tab.binom[nzB * kBinN + f], P6 = pw[5 * kT1PowRow + nzB - f];
                                    const double factor = C5 * C6 * P1 * P2 * P3 * P4 * P5 * P6;
                                    if (fabs(factor) < 1e-13) continue;
#pragma unroll
                                    for (int c = 0; c < kT1Group; c++) chi[c] = rn_add(chi[c], rn_mul(factor, row[c * nijk + f]));
                                }
                            }
                        }
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < kT1Group; c++)
                if (c < nj) scr[(int64_t)c * (nq + np) + nq + p] = skip[c] ? 0.0 : rn_mul(cc[c], chi[c]);
        }
    }
}

// contributions of a task's primitive pairs, added in their order
__global__ void t1_sum_kernel(Type1NumArgs a)
{
    for (int t = blockIdx.x; t < a.n_tasks; t += gridDim.x) {
        const int la = a.shell_L[a.task_a[t]], lb = a.shell_L[a.task_b[t]], np = ncart(la) * ncart(lb), nq = t1_nq(la + lb);
        const int nu = (int)(a.unit_off[t + 1] - a.unit_off[t]);
        const double *scr = a.scratch + a.scr_off[t] + nq;
        for (int p = threadIdx.x; p < np; p += blockDim.x) {
            double v = 0.0;
            for (int j = 0; j < nu; j++) v = rn_add(v, scr[(int64_t)j * (nq + np) + p]);
            a.out[a.out_off[t] + p] = v;
        }
    }
}

}  // namespace grpp

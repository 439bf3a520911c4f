// Host-built tables of the type 1 kernel (mmd.cuh): Cartesian pair tables, update programs and
// batch sizes per (la, lb).
#pragma once

#include <algorithm>
#include <utility>
#include <vector>

#include "mmd.cuh"

namespace grpp {

// Cartesian pair table of one (bra, ket) table class for mmd_kernel, pairs of equal loop counts
// (tx, uy) side by side so that the lanes of a warp run equal contractions.
static void mmd_pair_table(const int8_t *ca, int la, const int8_t *cb, int lb, std::vector<int4> &out)
{
    const int nA = ncart(la), nB = ncart(lb), S = la + lb, lb1 = lb + 1, nax = mmd_e_axis(la, lb), nos = (la + 1) * lb1;
    std::vector<int> xbase((la + 1) * lb1);
    for (int az = 0, o = 0; az <= la; az++)
        for (int bz = 0; bz <= lb; bz++) {
            const int W = S - az - bz;
            xbase[az * lb1 + bz] = o;
            o += (W + 1) * (W + 2) / 2;
        }
    std::vector<std::pair<int, int4>> rows;
    for (int m = 0; m < nA; m++)
        for (int n = 0; n < nB; n++) {
            const int8_t *a = ca + 3 * m, *b = cb + 3 * n;
            const int W = S - a[2] - b[2];
            // rows of X have t + u <= W: exponents that add up to L meet this with equality
            const int tx = std::min(a[0] + b[0], W), uy = std::min(a[1] + b[1], W - tx);
            const int4 r = mmd_pair(mmd_e_row(lb, a[0], b[0]), nax + mmd_e_row(lb, a[1], b[1]), xbase[a[2] * lb1 + b[2]], W,
                                    tx, uy, a[0] * lb1 + b[0], nos + a[1] * lb1 + b[1], 2 * nos + a[2] * lb1 + b[2], m * nB + n);
            rows.push_back({((tx * 32 + uy) * 16 + a[2]) * 16 + b[2], r});
        }
    std::stable_sort(rows.begin(), rows.end(), [](const std::pair<int, int4> &x, const std::pair<int, int4> &y) { return x.first > y.first; });
    for (auto &r : rows) out.push_back(r.second);
}

// Update programs and batch sizes of mmd_kernel for every la, lb <= kMmdMaxL.
struct MmdTables {
    std::vector<MmdClass> classes;
    std::vector<int> levels;
    std::vector<int2> etab, otab, rtab, ztab;
};

static void mmd_build_classes(MmdTables &T)
{
    // R^n_tuv programs per S: level s holds n = 0..S-s, entries (t, u, v) in level order
    std::vector<int> r_off(2 * kMmdMaxL + 1, 0), maxlev(2 * kMmdMaxL + 1, 1);
    std::vector<std::vector<int>> r_lv(2 * kMmdMaxL + 1);
    for (int S = 0; S <= 2 * kMmdMaxL; S++) {
        r_off[S] = (int)T.rtab.size();
        r_lv[S].push_back(0);
        maxlev[S] = S + 1;
        for (int s = 1; s <= S; s++) {
            r_lv[S].push_back((int)T.rtab.size() - r_off[S]);
            const int ne = (s + 1) * (s + 2) / 2, ne1 = s * (s + 1) / 2, ne2 = (s - 1) * s / 2;
            maxlev[S] = std::max(maxlev[S], ne * (S - s + 1));
            for (int n = 0; n <= S - s; n++)
                for (int idx = 0; idx < ne; idx++) {
                    int kk = 0;
                    while ((kk + 1) * (kk + 2) / 2 <= idx) kk++;
                    const int v = idx - kk * (kk + 1) / 2, u = kk - v, t = s - kk;
                    // step down along z if t = u = 0, else along y if t = 0, else along x
                    int uu = u, vv = v, kq, ax;
                    if (t + u == 0) {
                        vv = v - 1;
                        kq = v;
                        ax = 2;
                    } else if (t == 0) {
                        uu = u - 1;
                        kq = u;
                        ax = 1;
                    } else {
                        kq = t;
                        ax = 0;
                    }
                    // the entry takes order n (1/r^2 terms) and n + 1 of the levels s-1, s-2
                    const int src1 = n * ne1 + r_in_level(uu, vv);
                    const int src2 = kq > 1 ? n * ne2 + r_in_level(uu == u ? u : u - 2, vv == v ? v : v - 2) : 0;
                    T.rtab.push_back(mmd_r_code(src1, src2, n == 0 ? r0_row(S, t, u) + v : kMmdNoR0, kq, ax));
                }
        }
        r_lv[S].push_back((int)T.rtab.size() - r_off[S]);
    }
    for (int la = 0; la <= kMmdMaxL; la++)
        for (int lb = 0; lb <= kMmdMaxL; lb++) {
            MmdClass c{};
            const int S = la + lb, lb1 = lb + 1, nax = mmd_e_axis(la, lb), nos = (la + 1) * lb1;
            c.la = la;
            c.lb = lb;
            c.S = S;
            c.nE = 3 * nax;
            c.nR0 = mmd_tet(S);
            c.maxlev = maxlev[S];
            c.e_off = (int)T.etab.size();
            c.o_off = (int)T.otab.size();
            c.z_off = (int)T.ztab.size();
            c.r_off = r_off[S];
            std::vector<int> el, ol;
            for (int w = 0; w <= S; w++) {
                el.push_back((int)T.etab.size() - c.e_off);
                ol.push_back((int)T.otab.size() - c.o_off);
                if (w == 0) continue;  // E[ax][0][0][0] = S[ax][0][0] = K[ax]: set with the scalars
                for (int ax = 0; ax < 3; ax++)
                    for (int i = std::max(0, w - lb); i <= std::min(la, w); i++) {
                        const int j = w - i, e000 = ax * nax, row = e000 + mmd_e_row(lb, i, j);
                        // t = 0 steps down in j if i = 0, else in i; t >= 1 takes both rows
                        const int ri = i > 0 ? e000 + mmd_e_row(lb, i - 1, j) : e000, rj = j > 0 ? e000 + mmd_e_row(lb, i, j - 1) : e000;
                        T.etab.push_back(mmd_e_code0(row, i > 0 ? ri : rj, ax, i > 0 ? 0 : 1, w > 1));
                        for (int t = 1; t <= w; t++)
                            T.etab.push_back(mmd_e_code(row + t, i > 0 ? ri + t - 1 : e000, j > 0 ? rj + t - 1 : e000, ax, i, j, t));
                        const int o000 = ax * nos;
                        auto o = [&](int ii, int jj) { return o000 + ii * lb1 + jj; };
                        if (i == 0)
                            T.otab.push_back(mmd_o_code(o(0, j), o(0, j - 1), j > 1 ? o(0, j - 2) : o000, o000, j - 1, 0, ax, 1));
                        else
                            T.otab.push_back(mmd_o_code(o(i, j), o(i - 1, j), i > 1 ? o(i - 2, j) : o000,
                                                        j > 0 ? o(i - 1, j - 1) : o000, i - 1, j, ax, 0));
                    }
            }
            el.push_back((int)T.etab.size() - c.e_off);
            ol.push_back((int)T.otab.size() - c.o_off);
            for (int az = 0; az <= la; az++)
                for (int bz = 0; bz <= lb; bz++)
                    for (int t = 0; t <= S - az - bz; t++)
                        for (int u = 0; u <= S - az - bz - t; u++)
                            T.ztab.push_back(mmd_z_code(r0_row(S, t, u), 2 * nax + mmd_e_row(lb, az, bz), az + bz));
            c.nX = (int)T.ztab.size() - c.z_off;
            c.lv = (int)T.levels.size();
            T.levels.insert(T.levels.end(), el.begin(), el.end());
            T.levels.insert(T.levels.end(), ol.begin(), ol.end());
            T.levels.insert(T.levels.end(), r_lv[S].begin(), r_lv[S].end());
            // triples per batch: as many as the block's shared memory holds
            for (int kind = 0; kind < 2; kind++)
                for (int lg = 1; lg <= kMmdMaxLgT; lg++) {
                    MmdClass x = c;
                    x.lgT[kind] = lg;
                    if (mmd_smem_doubles(x) * (int)sizeof(double) <= kMmdSmem) c.lgT[kind] = lg;
                }
            T.classes.push_back(c);
        }
}

// Supported angular momenta of one batch's type 1 and overlap items: lmax the largest L, smax the largest
// L_A + L_B. Every pair up to i shells; one L = 7 shell with L_A + L_B <= 11, L = 8 with L_A + L_B <= 8. Every
// class within these fits kMmdSmem.
static bool mmd_accepts(int lmax, int smax) { return lmax <= 6 || (lmax == 7 && smax <= 11) || (lmax == kMmdMaxL && smax <= 8); }

}  // namespace grpp

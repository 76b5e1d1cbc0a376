// emu_apart.cpp -- TEST INFRASTRUCTURE: the two-launch step of small patches
// (k_records, then k_tile_apart) on the host: the records with their tile
// marks, then every marked tile's phases in the kernel's order with both
// sweeps' buffers side by side, the others' zeros. Not a product path.
#include <stdint.h>
#include <string.h>
#include <vector>
#include "../../dclaw_b200/csrc/tile.cuh"

using namespace dclaw;

template <int TX, int TY>
static int run(const dclaw_params* P, int mx, int my, double dx, double dy, double* q, const double* b, int nsteps,
               double dt_initial, double* dt_hist, double* cfl_hist) {
    using TG = TileGeom<TX, TY>;
    const Geom g{mx, my, mx + 4, my + 4, dx, dy};
    const size_t npad = (size_t)(mx + 4) * (my + 4), plane = (size_t)mx * my;
    const int ntx = (mx + TX - 1) / TX, nty = (my + TY - 1) / TY;
    // nothing is read that was not written: every buffer starts as NaN
    const double junk = 0.0 / 0.0;
    std::vector<double> rec(NREC * npad, junk), sm(TG::SMEM2_DOUBLES, junk);
    std::vector<uint32_t> bits(2 * (size_t)TG::NA);
    std::vector<char> flag((size_t)ntx * nty);
    const Rec R{rec.data(), npad};
    // k_tile_apart's split of its shared memory
    TileMem M[2];
    for (int dir = 0; dir < 2; ++dir) {
        M[dir].A = sm.data() + (size_t)dir * NW * TG::NA;
        M[dir].B = sm.data() + (size_t)2 * NW * TG::NA;
        M[dir].C = M[dir].B + (size_t)10 * TG::NB;
        M[dir].D = M[dir].C + (size_t)10 * TG::NC;
        M[dir].H = M[dir].D + (size_t)10 * TG::ND;
        M[dir].Bd = M[dir].H + TG::NHB;
        M[dir].T5 = nullptr;
        M[dir].Fy = M[dir].Bd + TG::NHB;
        M[dir].bits = bits.data() + (size_t)dir * TG::NA;
        M[dir].NA = TG::NA;
        M[dir].hw = TG::HW;
        M[dir].hv = TX + 6;
        if (M[dir].Fy + (size_t)10 * TG::NTS > sm.data() + sm.size()) return -2;
    }
    const double crit = critical_root(*P);
    std::vector<double> qa(q, q + 5 * plane), qb(5 * plane);
    double dt = dt_initial;
    for (int n = 0; n < nsteps; ++n) {
        int status = 0;
        std::fill(flag.begin(), flag.end(), 0);
        for (int j = -1; j <= my + 2; ++j)
            for (int i = -1; i <= mx + 2; ++i) {
                if (cell_record(*P, g, qa.data(), b, R, i, j)) status = DCLAW_ERR_NAN;
                if (!(R.get(R_H, pidx(g, i, j)) > 0.0)) continue;
                for (int t = 0; t < ntx * nty; ++t) {
                    const int i0 = 1 + t % ntx * TX, j0 = 1 + t / ntx * TY;
                    if (i >= i0 - 3 && i <= i0 + TX + 2 && j >= j0 - 3 && j <= j0 + TY + 2) flag[t] = 1;
                }
            }
        if (status) return status;
        std::fill(qb.begin(), qb.end(), junk);
        const double dtd[2] = {dt / dx, dt / dy};
        double cfl = 0.0;
        for (int t = 0; t < ntx * nty; ++t) {
            const int i0 = 1 + t % ntx * TX, j0 = 1 + t / ntx * TY;
            if (!flag[t]) {
                for (int j = j0; j < j0 + TY && j <= my; ++j)
                    for (int i = i0; i < i0 + TX && i <= mx; ++i)
                        for (int m = 0; m < 5; ++m) qb[(size_t)m * plane + (size_t)(j - 1) * mx + (i - 1)] = 0.0;
                continue;
            }
            std::fill(sm.begin(), sm.end(), junk);
            for (int dir = 0; dir < 2; ++dir) {
                M[dir].hi0 = i0 - 3;
                M[dir].hj0 = j0 - 3;
            }
            for (int it = 0; it < TG::NHB; ++it) tile_stage_hb(g, R, b, M[0], it);
            for (int dir = 0; dir < 2; ++dir)
                for (int it = 0; it < (dir == 0 ? TG::NXW : TG::NYW); ++it) {
                    bool ok;
                    const double s = tile_riemann(*P, g, R, M[dir], dir, it, i0, j0, TX, TY, ok, crit);
                    if (ok) cfl = fmax2(cfl, dtd[dir] * s);
                }
            // y first: neither sweep's fluxes read the other's
            for (int dir = 1; dir >= 0; --dir) {
                const int nsl = dir == 0 ? TY + 2 : TX + 2, span = dir == 0 ? TX : TY;
                const int smax = dir == 0 ? my + 1 : mx + 1, amax = dir == 0 ? mx : my, a0 = dir == 0 ? i0 : j0;
                for (int sl = 0; sl < nsl; ++sl) {
                    const int s = (dir == 0 ? j0 : i0) - 1 + sl;
                    if (s < 0 || s > smax) continue;
                    std::vector<double> v(15 * (size_t)(span + 1), 0.0);
                    for (int k = 0; k <= span && a0 + k <= amax + 1; ++k) {
                        if (dir == 0) tile_x_iface<TX, TY>(*P, M[0], s, a0 + k, i0, j0, dtd[0], &v[15 * k], nullptr);
                        else tile_y_iface<TX, TY>(*P, M[1], s, a0 + k, i0, j0, dtd[1], &v[15 * k], nullptr);
                    }
                    for (int k = 0; k < span && a0 + k <= amax; ++k) {
                        const int c = dir == 0 ? a0 + k : s, r = dir == 0 ? s : a0 + k;
                        tile_flux_cell<TX, TY, true>(*P, g, R, M[dir], dir, c, r, i0, j0, dtd[dir], &v[15 * k],
                                                     &v[15 * (k + 1)], 0, 0, nullptr);
                    }
                }
            }
            for (int it = 0; it < TX * TY; ++it)
                if (tile_final<TX, TY, true, true>(*P, g, R, M[it & 1], it, i0, j0, dt, dtd[0], dtd[1], qb.data()))
                    status = DCLAW_ERR_NAN;
        }
        if (status) return status;
        qa.swap(qb);
        dt_hist[n] = dt;
        cfl_hist[n] = cfl;
        dt = tick_next_dt(*P, dt, cfl);
    }
    memcpy(q, qa.data(), sizeof(double) * 5 * plane);
    return 0;
}

extern "C" int emu_run_apart(const dclaw_params* P, int mx, int my, double dx, double dy, double* q, const double* b,
                             int nsteps, double dt_initial, double* dt_hist, double* cfl_hist, int tx, int ty) {
    if (tx == 7 && ty == 7) return run<7, 7>(P, mx, my, dx, dy, q, b, nsteps, dt_initial, dt_hist, cfl_hist);
    if (tx == 14 && ty == 13) return run<14, 13>(P, mx, my, dx, dy, q, b, nsteps, dt_initial, dt_hist, cfl_hist);
    return -1;
}

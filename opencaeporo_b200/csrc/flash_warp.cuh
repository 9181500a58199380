// flash_warp.cuh -- PhaseSplit's restart loop on one warp per cell, for the
// few cells whose split keeps restarting (near-critical mixtures whose
// successive substitution converges over tens of thousands of iterations).
//
// Such a cell is a chain of tens of thousands of dependent iterations, so
// its time is latency: a dependent FP64 operation costs 8 cycles, a division
// 111 on one thread (72 as div_core), a logarithm 260, acos + cos 450. The
// operations of an iteration that are independent of one another run on
// different lanes and are exchanged through shared memory:
//   * Rachford-Rice: lane i forms component i's residual term, lane 16 + i
//     its Jacobian term; the sums are then taken on every lane in the
//     reference's order;
//   * compositions, fugacity ratios, K and the mixing rule's rows: one
//     component per lane;
//   * fugacities: phase 0 on lanes 0-15 and phase 1 on lanes 16-31 at once;
//     within a half, lanes 0-2 polish the three roots of the cubic; then
//     CalFugPhi's logarithms and reciprocals for the smallest and the largest
//     root and the pieces of the choice between them are formed side by side.
// Lanes that form different pieces run the same instructions on operands
// chosen per lane: different functions on different lanes of a warp would
// run one after another. All lanes take the same branches.
// Measured for 6 components, cycles per substitution step with 2.1 / 4.9 /
// 9.0 Rachford-Rice steps in it: 5,020 / 6,480 / 8,700 with the whole state
// on every lane and shuffles, 4,050 / 4,960 / 6,300 so; the 1M-cell block's
// fresh flash 157 -> 133 ms, four fluids of 8,192 wide states 555 -> 393 ms.
// Each value is formed by the same expression as in the one-thread form;
// the two agree to rounding (the compiler fuses multiply-adds per kernel), so
// an iteration count that ends on a convergence threshold can differ by a
// step.
#pragma once

#include "flash_cell.cuh"

namespace ocpf {

constexpr unsigned WARP_ALL = 0xffffffffu;

template <int NC>
struct WarpSplit {
    static constexpr bool LANES = NC <= 9;  // split_ssm2's form
    static_assert(NC <= 16, "one half-warp per phase holds at most 16 components");
    CellFlash<NC>& f;
    const int      lane, half, q;
    const unsigned hmask;
    double* xch;       // two exchange buffers of a lane's value each
    mutable int flip;  // which one the next exchange takes

    __device__ __forceinline__ explicit WarpSplit(CellFlash<NC>& cell)
        : f(cell),
          lane(threadIdx.x & 31),
          half((threadIdx.x & 31) >> 4),
          q(threadIdx.x & 15),
          hmask(((threadIdx.x & 31) >> 4) ? 0xffff0000u : 0x0000ffffu)
    {
        __shared__ __align__(16) double xbuf[4][64];
        xch  = xbuf[threadIdx.x >> 5];
        flip = 0;
    }

    // component q's entry of a per-component register array
    __device__ __forceinline__ double pick(const double* v) const
    {
        double r = v[0];
#pragma unroll
        for (int i = 1; i < NC; i++)
            if (q == i) r = v[i];
        return r;
    }

    // Puts every lane's value where all lanes of the warp can read it: the
    // buffer with lane l's value at [l], until the exchange after next. (A
    // value on all lanes takes one wide load per two values here, two
    // shuffles per value otherwise.)
    __device__ __forceinline__ const double* exchange(double mine) const
    {
        double* b = xch + flip;
        flip ^= 32;
        b[lane] = mine;
        __syncwarp();
        return b;
    }
    // v[i] = b[i]
    __device__ __forceinline__ void read(const double* b, double (&v)[NC]) const
    {
#pragma unroll
        for (int i = 0; i < NC; i += 2) {
            const double2 t = *reinterpret_cast<const double2*>(b + i);
            v[i]            = t.x;
            if (i + 1 < NC) v[i + 1] = t.y;
        }
    }
    // v[i] = lane i's value of the caller's half, on every lane of it
    __device__ __forceinline__ void gather(double mine, double (&v)[NC]) const
    {
        read(exchange(mine) + (half << 4), v);
    }

    // RachfordRice2, src/MixtureComp.cpp:1907-1959 (CellFlash::rachford_rice2)
    // for lane-resident K and z (component q's, the same in both halves;
    // lanes beyond NC repeat component 0), in two parts: the bracket, which
    // needs only K, and the Newton iteration.
    //
    // With all K within 2^-100 .. 2^100 and each z zero or within
    // 2^-300 .. 2^100 (`mid`), no operand of the iteration's divisions leaves
    // div_core's range, so it needs no range tests (a term's divisor that
    // cancels to zero makes the sums NaN instead of infinite, and the step
    // falls back to the bracket's lower half all the same): 610 -> 320 cycles
    // a turn. A divisor that div_core does not take (div_ones) sends the
    // whole iteration to the general form afterwards.
    struct Bracket {
        double numin, numax;
        bool   mid;
    };
    __device__ __forceinline__ Bracket rr_bracket(double K, bool zok) const
    {
        double ext = K;  // max K on half 0, min K on half 1
#pragma unroll
        for (int o = 1; o < NC; o *= 2) {
            const double v = __shfl_xor_sync(WARP_ALL, ext, o);
            ext            = (half ? v < ext : v > ext) ? v : ext;
        }
        const double bound = div1(1.0, 1 - ext);
        Bracket      br;
        br.mid   = __all_sync(WARP_ALL, zok && ext > 0x1p-100 && ext < 0x1p100);
        br.numin = __shfl_sync(WARP_ALL, bound, 0);
        br.numax = __shfl_sync(WARP_ALL, bound, 16);
        return br;
    }
    // Lane i forms component i's residual term, lane 16 + i its Jacobian
    // term; the sums run on every lane in the reference's order. The Newton
    // step is divided out ahead of the convergence test. Returns nu_0, and
    // in tmp 1 + nu_0 (K_q - 1).
    template <bool MID>
    __device__ __forceinline__ double rr_newton(double K, double z, const Bracket& br, int& it_rr) const
    {
        const double numin = br.numin, numax = br.numax;
        double       v = 0.5 * (numin + numax);
        // loop-invariant parts of component q's terms, formed as the
        // one-thread form forms them: z km1 / tmp and z km1 km1 / (tmp tmp)
        const double km1 = K - 1;
        const double zk  = z * km1;
        const double num = half ? zk * km1 : zk;
        const double tol = f.F.rr_tol;
        const int    cap = f.F.rr_maxit;
        int          iter = 0;
        bool         ones = false;
        while (true) {
            const double tmp  = 1 + v * km1;
            const double den  = tmp * (half ? tmp : 1.0);  // operand chosen, not path
            const double term = MID ? div_core(num, den) : div_slow(num, den);
            const double* xb = exchange(term);
            double        tr[NC], tj[NC], rj = 0, J = 0;
            read(xb, tr);
            read(xb + 16, tj);
#pragma unroll
            for (int i = 0; i < NC; i++) {
                rj += tr[i];
                J -= tj[i];
            }
            ones |= MID && (div_ones(den) || div_ones(J));
            const double dnuj = MID ? div_core(-rj, J) : div_slow(-rj, J);
            if (fabs(rj) < tol || iter > cap) break;
            const double tmpnu = v + dnuj;
            if (tmpnu < numax && tmpnu > numin)
                v = tmpnu;
            else if (dnuj > 0)
                v = (v + numax) / 2;
            else
                v = (v + numin) / 2;
            iter++;
        }
        if (MID && __any_sync(WARP_ALL, ones)) return rr_newton<false>(K, z, br, it_rr);
        it_rr += iter;
        return v;
    }

    // component q's row of 1 - k_ik, sqrt(A_q) and B_q; and the coefficients
    // of b in the two factors of the numerator and of the denominator of the
    // piece that lane q forms in fug_lane:
    //   q = 0, 4 (smallest, largest root)  (z - b) / 1
    //       1, 5                           (z + d1 b) / (z + d2 b)
    //       2, 3                           1 / b, 1 / a
    //       8                              (zmin - b) / (zmax - b)
    //       9                              (zmin + d1 b)(zmax + d2 b) / ((zmin + d2 b)(zmax + d1 b))
    //       10                             a / ((d2 - d1) b)
    // (other lanes repeat these), as fug_piece and gibbs_piece form them:
    // x - b is fma(-1, b, x), and a product by one changes nothing.
    struct LaneConst {
        double omb[NC], sA, Bi, sAk[NC], Bk[NC];
        double n1, n2, d1, d2;
        int    role;
    };
    __device__ __forceinline__ LaneConst lane_const() const
    {
        LaneConst c;
        const int row = q < NC ? q : 0;
#pragma unroll
        for (int k = 0; k < NC; k++) {
            c.omb[k] = f.F.omb[row * MAXNC + k];
            c.sAk[k] = f.sA[k];
            c.Bk[k]  = f.Bi[k];
        }
        c.sA = pick(f.sA);
        c.Bi = pick(f.Bi);
        c.role        = q < 8 ? q : 8 + (q & 3);
        const int  k  = c.role & 3;
        const bool gib = c.role >= 8;
        if (gib && k == 3) c.role = 10;
        c.n1 = k == 0 ? -1.0 : (k == 1 ? D1 : 0.0);
        c.n2 = gib && k == 1 ? D2 : 0.0;
        c.d1 = k == 0 ? (gib ? -1.0 : 0.0) : (k == 1 ? D2 : (gib ? D2 - D1 : (k == 2 ? 1.0 : 0.0)));
        c.d2 = gib && k == 1 ? D1 : 0.0;
        return c;
    }

    // One phase of CalFugPhi (src/MixtureComp.cpp:993-1101) on each half:
    // half j holds phase j's composition xj; returns phi of component q (lanes
    // beyond NC: of component 0) of phase `half` and leaves the phase's a, b and Z on every lane of the
    // half. Within a half, lanes 0-2 polish the cubic's roots; then one
    // division and one logarithm per lane form, side by side, CalFugPhi's
    // pieces for the smallest root (lanes 0-3), for the largest (4-7) and
    // the pieces of the choice between the two (8-10).
    template <bool FIXED>
    __device__ __forceinline__ double fug_lane(const double (&xj)[NC], const LaneConst& lc, double& aj, double& bj,
                                               double& zj) const
    {
        // mix_ab with row q's sum on lane q
        double s = 0, t[NC];
#pragma unroll
        for (int k = 0; k < NC; k++) s += lc.omb[k] * (lc.sAk[k] * xj[k]);
        const double tq = lc.sA * s;
        gather(tq, t);
        aj = 0;
        bj = 0;
#pragma unroll
        for (int i = 0; i < NC; i++) {
            aj += xj[i] * t[i];
            bj += lc.Bk[i] * xj[i];
        }
        const int  base = half << 4;
        double     zmin, zmax;
        const bool three = root_pair_group<FIXED>(aj, bj, hmask, base, q, zmin, zmax);
        __syncwarp();
        // num = (n1 b + u1) (n2 b + u2), den = (d1 b + w1) (d2 b + w2) with
        // the coefficients of the lane's piece (LaneConst); a factor that a
        // piece does not have is 0 b + 1
        const double z   = (lc.role & 4) ? zmax : zmin;
        const bool   gib = lc.role >= 8;
        const int    k   = lc.role & 3;
        const double u1  = k <= 1 ? z : (gib ? aj : 1.0);
        const double u2  = gib && k == 1 ? zmax : 1.0;
        const double w1  = k == 0 ? (gib ? zmax : 1.0) : (k == 1 ? z : (k == 2 ? 0.0 : aj));
        const double w2  = gib && k == 1 ? zmax : 1.0;
        const double num = fma(lc.n1, bj, u1) * fma(lc.n2, bj, u2);
        const double den = fma(lc.d1, bj, w1) * fma(lc.d2, bj, w2);
        const double d   = div1(num, den);
        const double ld    = log(d);
        const double piece = k <= 1 ? ld : d;
        int          from  = base;
        zj                 = zmin;
        const double g1 = __shfl_sync(WARP_ALL, piece, base + 8);
        const double g2 = __shfl_sync(WARP_ALL, piece, base + 9);
        const double gk = __shfl_sync(WARP_ALL, piece, base + 10);
        if (three) {
            zj = pick_root_from(zmin, zmax, g1, g2, gk);
            if (!(zj == zmin)) from += 4;
        }
        const double L1  = __shfl_sync(WARP_ALL, piece, from);
        const double L2  = __shfl_sync(WARP_ALL, piece, from + 1);
        const double ib  = __shfl_sync(WARP_ALL, piece, base + 2);
        const double ia  = __shfl_sync(WARP_ALL, piece, base + 3);
        const double cf  = div_const(aj, D1MD2, RCPD1MD2) * ib;
        const double zm1 = zj - 1;
        return phi_term_of<FIXED>(lc.Bi * ib, tq, ia, zm1, L1, cf, L2);
    }

    // One phase of CalFugPhi (src/MixtureComp.cpp:993-1101) on each half:
    // half j holds phase j's composition xj; returns phi of component q of
    // phase `half` and leaves the phase's a, b and Z on every lane of the
    // half. Within a half, lanes 0-2 polish the cubic's roots and lanes 0-3
    // form the two logarithms and two reciprocals.
    __device__ __forceinline__ double fug_lane_nr(const double* xj, double& aj, double& bj, double& zj) const
    {
        double t[NC];
        mix_ab<NC>(f.F, f.sA, f.Bi, xj, t, aj, bj);
        zj              = sol_eos_group(aj, bj, hmask, half << 4, q);
        const int    base  = half << 4;
        const double piece = fug_piece(q < 4 ? q : 3, zj, aj, bj);
        const double L1  = __shfl_sync(WARP_ALL, piece, base);
        const double L2  = __shfl_sync(WARP_ALL, piece, base + 1);
        const double ib  = __shfl_sync(WARP_ALL, piece, base + 2);
        const double ia  = __shfl_sync(WARP_ALL, piece, base + 3);
        const double cf  = div_const(aj, D1MD2, RCPD1MD2) * ib;
        const double zm1 = zj - 1;
        double       tq = 0, bq = 0;
#pragma unroll
        for (int i = 0; i < NC; i++) {
            if (q == i) {
                tq = t[i];
                bq = f.Bi[i];
            }
        }
        return q < NC ? phi_term(bq * ib, tq, ia, zm1, L1, cf, L2) : 0.0;
    }

    // The state of both phases on every lane from the per-lane pieces: a, b,
    // Z from lanes 0 and 16, phi_ji from lane 16 j + i, and f = phi x P.
    __device__ __forceinline__ void share_phases(double ph, double aj, double bj, double zj)
    {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            f.Aj[j] = __shfl_sync(WARP_ALL, aj, 16 * j);
            f.Bj[j] = __shfl_sync(WARP_ALL, bj, 16 * j);
            f.Zj[j] = __shfl_sync(WARP_ALL, zj, 16 * j);
#pragma unroll
            for (int i = 0; i < NC; i++) {
                const double p = __shfl_sync(WARP_ALL, ph, 16 * j + i);
                f.phi[j][i]    = p;
                f.fug[j][i]    = p * f.x[j][i] * f.P;
            }
        }
    }

    // CalFugPhiAll for NP = 2 (src/MixtureComp.cpp:1103-1145) from f.x.
    __device__ __forceinline__ void fug_phi_all()
    {
        double xj[NC];
#pragma unroll
        for (int k = 0; k < NC; k++) xj[k] = half ? f.x[1][k] : f.x[0][k];
        double aj, bj, zj;
        const double ph = fug_lane_nr(xj, aj, bj, zj);
        share_phases(ph, aj, bj, zj);
    }

    // SplitSSM2's iterations with UpdateXRR, src/MixtureComp.cpp:1881-1902,
    // 2030-2043, from f.Ks while Se exceeds Stol, `iter` steps already taken;
    // f.ssmsp_conflag falls when the cap ends them. Inside the loop lane
    // (j, i) holds component i's K and z and its x_ji and phi_ji; the state
    // goes to every lane after the last step. Returns Se. FIXED:
    // PrCubic::Fixed's roundings, the one-lane kernel's (sp_ssm_body).
    template <bool FIXED>
    __device__ __forceinline__ double ssm_steps(double Se, double Stol, int maxIt, int& iter)
    {
        double       K    = pick(f.Ks), x1 = 0, x0 = 0, ph = 0, aj = 0, bj = 0, zj = 0;
        const double    z = pick(f.zi), P = f.P;
        double          nu0   = f.nu[0];
        int             it_rr = 0;
        const int       iter0 = iter;
        const bool      zok = __all_sync(WARP_ALL, z == 0 || (z > 0x1p-300 && z < 0x1p100));
        const LaneConst lc  = lane_const();
        while (Se > Stol) {
            const Bracket br = rr_bracket(K, zok);
            nu0 = br.mid ? rr_newton<true>(K, z, br, it_rr) : rr_newton<false>(K, z, br, it_rr);
            // UpdateXRR
            x1 = div1(z, 1 + nu0 * (K - 1));
            x0 = K * x1;
            double xj[NC];
            gather(half ? x1 : x0, xj);
            ph = fug_lane<FIXED>(xj, lc, aj, bj, zj);
            // lane i: component i's squared fugacity-ratio residual; lane
            // 16 + i: its new K (one division on every lane)
            const double fg   = ph * (half ? x1 : x0) * P;
            const double recv = __shfl_xor_sync(WARP_ALL, half ? fg : ph, 16);
            const double quo  = div1(half ? ph : recv, half ? recv : fg);
            const double dq   = quo - 1, dq2 = dq * dq;
            K = __shfl_sync(WARP_ALL, quo, 16 + (q < NC ? q : 0));
            double r2[NC];
            read(exchange(dq2), r2);
            Se = 0;
#pragma unroll
            for (int i = 0; i < NC; i++) Se = __dadd_rn(Se, r2[i]);
            iter++;
            if (iter > maxIt) {
                f.ssmsp_conflag = false;
                break;
            }
        }
        if (iter > iter0) {
            f.nu[0] = nu0;
            f.nu[1] = 1 - nu0;
#pragma unroll
            for (int i = 0; i < NC; i++) {
                f.x[1][i] = __shfl_sync(WARP_ALL, x1, i);
                f.x[0][i] = __shfl_sync(WARP_ALL, x0, i);
                f.Ks[i]   = __shfl_sync(WARP_ALL, K, i);
            }
            share_phases(ph, aj, bj, zj);
        }
        f.it_rr += it_rr;
        return Se;
    }

    // SplitSSM2, src/MixtureComp.cpp:1847-1903 (CellFlash::split_ssm2)
    __device__ __forceinline__ void split_ssm2_lanes(bool restart)
    {
        f.ssmsp_conflag = true;
        double Se       = 1;
        double Stol     = f.F.ssmsp_tol2;
        int    maxIt    = f.F.ssmsp_maxit;
        if (restart) {
            Stol *= 1e-1;
            maxIt *= 2;
        }
        if (f.Yt < 1.1) {
            Stol *= 1e-1;
            maxIt *= 2;
        }
        int iter = 0;
        Se       = ssm_steps<false>(Se, Stol, maxIt, iter);
        f.ssmsp_realTol = sqrt(Se);
        f.it_ssmsp += iter;
    }

    // RachfordRice2, src/MixtureComp.cpp:1907-1959 (CellFlash::rachford_rice2):
    // lane i forms component i's residual term, lane 16 + i its Jacobian
    // term; the sums run on every lane in the reference's order.
    __device__ void rachford_rice2_all()
    {
        double Kmin = f.Ks[0], Kmax = f.Ks[0];
#pragma unroll
        for (int i = 1; i < NC; i++) {
            if (f.Ks[i] < Kmin) Kmin = f.Ks[i];
            if (f.Ks[i] > Kmax) Kmax = f.Ks[i];
        }
        const double bound = 1 / (1 - (half ? Kmin : Kmax));
        const double numin = __shfl_sync(WARP_ALL, bound, 0);
        const double numax = __shfl_sync(WARP_ALL, bound, 16);
        double       v     = 0.5 * (numin + numax);
        // loop-invariant parts of component q's terms, formed as the
        // one-thread form forms them: z km1 / tmp and z km1 km1 / (tmp tmp)
        const double km1 = pick(f.Ks) - 1;
        const double zk  = pick(f.zi) * km1;
        const double num = half ? zk * km1 : zk;
        int          iter = 0;
        while (true) {
            const double tmp  = 1 + v * km1;
            const double term = num / (half ? tmp * tmp : tmp);
            double       rj = 0, J = 0;
#pragma unroll
            for (int i = 0; i < NC; i++) {
                rj += __shfl_sync(WARP_ALL, term, i);
                J -= __shfl_sync(WARP_ALL, term, 16 + i);
            }
            if (fabs(rj) < f.F.rr_tol || iter > f.F.rr_maxit) break;
            const double dnuj  = -rj / J;
            const double tmpnu = v + dnuj;
            if (tmpnu < numax && tmpnu > numin)
                v = tmpnu;
            else if (dnuj > 0)
                v = (v + numax) / 2;
            else
                v = (v + numin) / 2;
            iter++;
        }
        f.it_rr += iter;
        f.nu[0] = v;
        f.nu[1] = 1 - v;
    }

    // UpdateXRR (src/MixtureComp.cpp:2030-2043): lane i forms x_1i and x_0i.
    __device__ __forceinline__ void update_x()
    {
        const double tmp = 1 + f.nu[0] * (pick(f.Ks) - 1);
        const double x1  = pick(f.zi) / tmp;
        const double x0  = pick(f.Ks) * x1;
#pragma unroll
        for (int i = 0; i < NC; i++) {
            f.x[1][i] = __shfl_sync(WARP_ALL, x1, i);
            f.x[0][i] = __shfl_sync(WARP_ALL, x0, i);
        }
    }

    // SplitSSM2 with UpdateXRR, src/MixtureComp.cpp:1847-1903, 2030-2043, every
    // lane holding the whole state between its pieces
    // (CellFlash::split_ssm2 with the pieces above).
    __device__ void split_ssm2_all(bool restart)
    {
        f.ssmsp_conflag = true;
        double Se       = 1;
        double Stol     = f.F.ssmsp_tol2;
        int    maxIt    = f.F.ssmsp_maxit;
        if (restart) {
            Stol *= 1e-1;
            maxIt *= 2;
        }
        if (f.Yt < 1.1) {
            Stol *= 1e-1;
            maxIt *= 2;
        }
        int iter = 0;
        while (Se > Stol) {
            rachford_rice2_all();
            update_x();
            fug_phi_all();
            // lane i: component i's squared fugacity-ratio residual; lane
            // 16 + i: its new K (one division on every lane)
            const double quo = (half ? pick(f.phi[1]) : pick(f.fug[1])) / (half ? pick(f.phi[0]) : pick(f.fug[0]));
            const double v   = half ? quo : sq(quo - 1);
            Se               = 0;
#pragma unroll
            for (int i = 0; i < NC; i++) {
                Se      = __dadd_rn(Se, __shfl_sync(WARP_ALL, v, i));
                f.Ks[i] = __shfl_sync(WARP_ALL, v, 16 + i);
            }
            iter++;
            if (iter > maxIt) {
                f.ssmsp_conflag = false;
                break;
            }
        }
        f.ssmsp_realTol = sqrt(Se);
        f.it_ssmsp += iter;
    }

    // The lane-resident loop, up to 9 components: a step takes 5,100-5,400
    // cycles instead of 6,900 (6 components, 5.7 Rachford-Rice steps). With 12,
    // SplitNR's code beside that loop compiles to other roundings than
    // before, which the chaotic restart chains amplify, so they keep the
    // loop whose state is on every lane.
    __device__ __forceinline__ void split_ssm2(bool restart)
    {
        if constexpr (LANES)
            split_ssm2_lanes(restart);
        else
            split_ssm2_all(restart);
    }

    // ln(f_1i / f_0i) of every component, one per lane, and their squared sum
    __device__ __forceinline__ double residual(double* res) const
    {
        const double r   = log(pick(f.fug[1]) / pick(f.fug[0]));
        double       eNR = 0;
#pragma unroll
        for (int i = 0; i < NC; i++) {
            res[i] = __shfl_sync(WARP_ALL, r, i);
            eNR += res[i] * res[i];
        }
        return eNR;
    }

    // CellFlash::sp_nr_update; a call of its own for 9 components, where its
    // code inlined beside the lane-resident loop spills and rounds differently
    __device__ __noinline__ double nr_update_call(double* res) { return f.sp_nr_update(res); }
    __device__ __forceinline__ double nr_update(double* res)
    {
        if constexpr (LANES && NC > 6)
            return nr_update_call(res);
        else
            return f.sp_nr_update(res);
    }

    // SplitNR, src/MixtureComp.cpp:2057-2166 (CellFlash::split_nr with the
    // pieces above; the Newton step itself runs on every lane).
    __device__ void split_nr()
    {
        f.nrsp_conflag = false;
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int i = 0; i < NC; i++) f.n[j][i] = f.nu[j] * f.x[j][i];
        double res[NC];
        double eNR        = sqrt(residual(res));
        const double eNR0 = eNR;
        int          iter = 0;
        while (eNR > f.F.nrsp_tol) {
            const double en = nr_update(res);
            fug_phi_all();
            eNR = sqrt(residual(res));
            iter++;
            if (eNR > eNR0 || iter > f.F.nrsp_maxit) break;
            if (en / (2 * NC) < 1e-8) {
                f.nrsp_conflag = true;
                break;
            }
        }
        f.nrsp_realTol = eNR;
        if (eNR < f.F.nrsp_tol) f.nrsp_conflag = true;
        f.it_nrsp += iter;
    }
};

}  // namespace ocpf

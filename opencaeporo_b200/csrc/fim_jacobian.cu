// fim_jacobian.cu -- the consumer of the flash's derivatives: the bulk part
// of the FIM Jacobian as IsoT_FIM::AssembleMatBulksNew builds it
// (src/OCPFluidMethod.cpp:1569-1840), and the upstream choice of every
// connection and phase that precedes it (src/BulkConn.cpp:170-215).
//
//   * k_upwind, one thread per (phase, connection): upstream bulk and mean
//     density;
//   * k_conn_block, one lane per connection, one warp per end and group of
//     rows: forms each entry of those rows of dF/dXp and dF/dXs and at once
//     multiplies it into the rows of dt (dF/dXp + dF/dXs dSec_dPri)
//     (DaABpbC, src/DenseMat.cpp:75-94), held in registers; stored as the
//     connection's off-diagonal blocks;
//   * k_diag_rows, one thread per (row, bulk): the accumulation block plus
//     every incident connection's diagonal contribution, gathered through a
//     per-bulk list in connection order, which is the order the reference's
//     AddDiag calls sum them in.
// Every operation is an explicitly rounded intrinsic in the reference's
// left-to-right expression order (x / 2 as x * 0.5, the same value); the dense product sums over k in order
// and adds the dF/dXp entry last, as dgemm with beta = 1 does.
#include <algorithm>
#include <cstring>
#include <new>
#include <vector>

#include <cuda_runtime.h>

#include "ocp_flash.h"

namespace ocpf {
namespace {

constexpr double J_CONV1 = 5.61458;      // include/OCPConst.hpp
constexpr double J_CONV2 = 1.12712E-3;   // Darcy constant, field units
constexpr double J_GRAV  = 0.00694444;   // GRAVITY_FACTOR
constexpr int    J_NP    = 3;

__device__ __forceinline__ double M(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double A(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double S(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double D(double a, double b) { return __ddiv_rn(a, b); }

struct ConnDev {
    int64_t        nb, nconn;
    const int64_t* bId;
    const int64_t* eId;
    const double*  area;
    const int64_t* adj_off;  // [nb + 1]
    const int64_t* adj;      // c + 1 at the begin bulk, -(c + 1) at the end bulk, c increasing
};

__global__ void __launch_bounds__(256) k_upwind(const ConnDev C, const ocpf_jac_bulk B, int32_t* up, double* uprho)
{
    const int64_t nc = C.nconn, nb = C.nb;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < J_NP * nc;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int     j = (int)(t / nc);
        const int64_t c = t - j * nc;
        const int64_t b = C.bId[c], e = C.eId[c];
        const bool    xb = B.phaseExist[j * nb + b] != 0, xe = B.phaseExist[j * nb + e] != 0;
        double        rho;
        if (xb && xe) {
            const double sb = B.S[j * nb + b], se = B.S[j * nb + e];
            rho = D(A(M(B.rho[j * nb + b], sb), M(B.rho[j * nb + e], se)), A(sb, se));
        } else if (xb) {
            rho = B.rho[j * nb + b];
        } else if (xe) {
            rho = B.rho[j * nb + e];
        } else {
            up[j * nc + c]    = (int32_t)b;
            uprho[j * nc + c] = 0;
            continue;
        }
        const double gr = M(J_GRAV, rho);
        const double dP = S(S(B.Pj[j * nb + b], M(gr, B.depth[b])), S(B.Pj[j * nb + e], M(gr, B.depth[e])));
        up[j * nc + c]    = (int32_t)(dP < 0 ? e : b);
        uprho[j * nc + c] = rho;
    }
}

// Work split of k_conn_block: a tile of 32 consecutive connections (one per
// lane) is served by 2 G warps, warp (end, g) forming NR of the NCOM rows of
// that end's block, all NCOL columns of them in registers; every dF/dXs entry
// is multiplied into them as it is formed, so that neither the dF/dXs rows
// nor the product's columns are stored in between. Lanes of a warp hold
// consecutive connections, whose end bulks are consecutive along a grid line:
// the dSec_dPri entries come as coalesced 256-byte lines. For 3 and 6
// components a tile's entries (both ends) are copied asynchronously into
// shared memory first, 61 KB for 6 components, three tiles an SM in flight.
//
// Bound by latency and the issue of ~4,000 unfused FP64 operations of a
// two-phase connection (FP64 pipe 37 % busy at 12 warps an SM), with ~1 KB of
// stores and 2 KB of loads beside them. 60 x 220 x 85 bulks, 6 components,
// whole call: 11.1 ms with the rows and columns through shared memory (one
// thread per row, then per column), 9.8 ms with this split reading dSec_dPri
// directly, 7.2 ms staged, 6.2 ms with the next composition's partials
// prefetched and the quotients batched (div_by). 3 components, 561,000 bulks:
// 3.47 -> 1.28 ms; 9 and 12 components, 100,000 bulks: 2.42 -> 1.46 and 6.76 ->
// 3.55 ms. Rows a thread: 4 for 3, 6 and 12 components, 5 for 9, where 3 or 4
// rows took 2.43 ms.
template <int NCOM>
struct ConnTile {
    static constexpr int NCOL  = NCOM + 1;
    static constexpr int NSEC  = 3 + 2 * (NCOM - 1);     // dSec_dPri rows of a two-phase bulk
    static constexpr int G     = NCOM <= 4 ? 1 : (NCOM <= 10 ? 2 : 4);  // row groups
    static constexpr int NR    = (NCOM + G - 1) / G;     // rows of a group; the last group may repeat some
    static constexpr int TILES = G == 1 ? 2 : 1;         // tiles per block
    static constexpr int TPT   = 64 * G;                 // threads per tile
    static constexpr int THREADS = TPT * TILES;
    static constexpr int MINB    = NCOM <= 7 ? 3 : (NCOM <= 10 ? 2 : 1);
    // dSec_dPri entries of both ends staged in shared memory
    static constexpr bool   STAGED  = NCOM <= 7;
    static constexpr int    NENT    = NSEC * NCOL;
    static constexpr size_t SEC     = STAGED ? (size_t)2 * NENT * 32 : 0;  // doubles per tile
};

// Per connection and phase, formed once per tile (stage_phase).
enum : int { Q_DP = 0, Q_XI, Q_MU, Q_Y, Q_MUP, Q_XIP, Q_RHOP, Q_RHOPB, Q_RHOPE, Q_TR, Q_COUNT };
// flag bits of a connection and phase; bits 8-15 and 16-23 hold the
// composition counts of the begin and end bulk
enum : uint32_t { F_EXU = 1, F_UPB = 2, F_EXB = 4, F_EXE = 8, F_SDB = 16, F_SDE = 32, F_BAD = 64, F_SAFE = 128 };

template <int NCOM>
struct ConnStage {
    double   sec[ConnTile<NCOM>::SEC + 1];
    double   x[J_NP * NCOM][32];  // xij of the upstream bulk
    double   q[J_NP][Q_COUNT][32];
    uint32_t f[J_NP][32];
};

// One 8-byte asynchronous copy into shared memory.
__device__ __forceinline__ void copy8(double* dst, const double* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// |x| within 2^-200 .. 2^200, or zero: a product of two such values divided
// by a third neither overflows nor loses bits to underflow on the way.
__device__ __forceinline__ bool mid_range(double x)
{
    const uint32_t h = (uint32_t)__double2hiint(x) & 0x7fffffffu;
    return (h - (823u << 20)) < (400u << 20) || x == 0;
}

__device__ __noinline__ double div_any(double a, double b) { return __ddiv_rn(a, b); }

// q[i] = a[i] / b, correctly rounded, from y = RN(1 / b) (P. Markstein,
// Computation of elementary functions on the IBM RISC System/6000 processor,
// 1990): one correction makes q faithful, its residual is then exact, and
// the second rounds correctly. All quotients by a phase's viscosity share y,
// and nothing orders them against one another. `safe`: a, b and a / b are
// away from the ends of the exponent range.
template <int N>
__device__ __forceinline__ void div_by(const double (&a)[N], double b, double y, bool safe, double (&q)[N])
{
#pragma unroll
    for (int i = 0; i < N; i++) {
        q[i] = M(a[i], y);
        q[i] = __fma_rn(__fma_rn(-b, q[i], a[i]), y, q[i]);
        q[i] = __fma_rn(__fma_rn(-b, q[i], a[i]), y, q[i]);
    }
    if (!safe)
        for (int i = 0; i < N; i++) q[i] = div_any(a[i], b);
}

template <int NCOM>
__device__ __forceinline__ void stage_phase(const ConnDev& C, const ocpf_jac_bulk& B, const int32_t* up,
                                            const double* uprho, int64_t c, int j, int lane, ConnStage<NCOM>& sm)
{
    const int64_t nc = C.nconn, nb = C.nb;
    const int64_t bId = C.bId[c], eId = C.eId[c];
    const int64_t u   = up[j * nc + c];
    const bool    xb  = B.phaseExist[j * nb + bId] != 0, xe = B.phaseExist[j * nb + eId] != 0;
    const uint32_t vB = B.pVnumCom[j * nb + bId], vE = B.pVnumCom[j * nb + eId];
    uint32_t       f  = (u == bId ? F_UPB : 0u) | (xb ? F_EXB : 0u) | (xe ? F_EXE : 0u) |
                 (B.pSderExist[j * nb + bId] != 0 ? F_SDB : 0u) | (B.pSderExist[j * nb + eId] != 0 ? F_SDE : 0u);
    // shapes a flash writes: at most NCOM - 1 compositions per phase (and
    // NSEC dSec_dPri rows, checked by the caller); anything else (and an
    // upstream bulk that is neither end) gives NaN blocks
    if ((u != bId && u != eId) || vB >= (uint32_t)NCOM || vE >= (uint32_t)NCOM)
        f |= F_BAD;
    else
        f |= vB << 8 | vE << 16;
    if (!(f & F_BAD) && (u == bId ? xb : xe)) {
        f |= F_EXU;
        for (int i = 0; i < NCOM; i++) copy8(&sm.x[j * NCOM + i][lane], B.xij + (int64_t)(j * NCOM + i) * nb + u);
        const int64_t uj     = j * nb + u;
        const double  Akd    = M(J_CONV1 * J_CONV2, C.area[c]);
        const double  dGamma = M(J_GRAV, S(B.depth[bId], B.depth[eId]));
        const double  mu = B.mu[uj], muP = B.muP[uj], t = M(Akd, B.kr[uj]);
        const double  y  = __drcp_rn(mu);
        if (mid_range(mu) && mu != 0 && mid_range(muP) && mid_range(t)) f |= F_SAFE;
        sm.q[j][Q_DP][lane] = S(S(B.Pj[j * nb + bId], B.Pj[j * nb + eId]), M(uprho[j * nc + c], dGamma));
        sm.q[j][Q_XI][lane]    = B.xi[uj];
        sm.q[j][Q_MU][lane]    = mu;
        sm.q[j][Q_Y][lane]     = y;
        sm.q[j][Q_MUP][lane]   = muP;
        sm.q[j][Q_XIP][lane]   = B.xiP[uj];
        sm.q[j][Q_RHOP][lane]  = B.rhoP[uj];
        sm.q[j][Q_RHOPB][lane] = xb ? B.rhoP[j * nb + bId] : 0.0;
        sm.q[j][Q_RHOPE][lane] = xe ? B.rhoP[j * nb + eId] : 0.0;
        const double num[1] = {t};
        double       tr[1];
        div_by(num, mu, y, (f & F_SAFE) != 0, tr);
        sm.q[j][Q_TR][lane] = tr[0];
    }
    sm.f[j][lane] = f;
}

// Rows row0 .. row0 + NR - 1 (of the NCOM component rows; those before
// `first` belong to the group before and are not stored) of one end's block: dF/dXp's column 0 and each dF/dXs entry in the reference's order,
// every entry multiplied into the NCOL sums as soon as it is formed. `end`
// is warp-uniform. The sum of an entry over k runs over the compact
// dSec_dPri rows in order, the dF/dXp entry last, as dgemm with beta = 1
// forms it; stored as (row eId, col bId) = -bmatB or (row bId, col eId) = bmatE.
template <int NCOM>
__device__ __forceinline__ void conn_rows(const ConnDev& C, const ocpf_jac_bulk& B, double dt,
                                          const ocpf_jac_out& O, int64_t c, int lane, int end, int row0, int first,
                                          const ConnStage<NCOM>& sm)
{
    using CT = ConnTile<NCOM>;
    constexpr int NCOL = CT::NCOL, NR = CT::NR;
    const int64_t nc = C.nconn, nb = C.nb;
    const int64_t bId = C.bId[c], eId = C.eId[c];
    const int64_t n      = end ? eId : bId;  // this end's bulk
    const double  Akd    = M(J_CONV1 * J_CONV2, C.area[c]);
    const double  dGamma = M(J_GRAV, S(B.depth[bId], B.depth[eId]));
    const int     vsh    = end ? 16 : 8;
    const uint32_t ex_me = end ? F_EXE : F_EXB, sd_me = end ? F_SDE : F_SDB;
    uint32_t      fl[J_NP];
    int           nsat = 0, ncomp = 0, noth = 0;
    bool          ok = true, odd = false;
#pragma unroll
    for (int j = 0; j < J_NP; j++) {
        fl[j] = sm.f[j][lane];
        nsat += (fl[j] & sd_me) ? 1 : 0;
        ncomp += (fl[j] >> vsh) & 0xff;
        noth += ((fl[j] >> (24 - vsh)) & 0xff) + ((fl[j] & (end ? F_SDB : F_SDE)) ? 1 : 0);
        ok  = ok && !(fl[j] & F_BAD);
        // a phase of both bulks with different composition counts (no flash
        // writes it): its columns can run into the next phase's
        odd = odd || ((fl[j] & F_EXB) && (fl[j] & F_EXE) && ((fl[j] >> 8) & 0xff) != ((fl[j] >> 16) & 0xff));
    }
    ok = ok && nsat + ncomp <= CT::NSEC && noth <= CT::NSEC;
    double* dst = (end ? O.offBE : O.offEB) + c;
    if (!ok) {
        for (int e = (row0 ? row0 + 1 : 0) * NCOL; e < (row0 + NR + 1) * NCOL; e++)
            dst[(int64_t)e * nc] = __longlong_as_double(0x7ff8000000000000LL);
        return;
    }
    if (row0 == 0) {
#pragma unroll
        for (int col = 0; col < NCOL; col++) dst[(int64_t)col * nc] = end ? M(0.0, dt) : -M(0.0, dt);
    }
    double acc[NR][NCOL], p[NR], rs[J_NP][NR];
#pragma unroll
    for (int i = 0; i < NR; i++) {
        p[i] = 0;
#pragma unroll
        for (int col = 0; col < NCOL; col++) acc[i][col] = 0;
#pragma unroll
        for (int j1 = 0; j1 < J_NP; j1++) rs[j1][i] = 0;
    }
    // dF/dXp's column 0 and the saturation columns of dF/dXs
    double dPc[J_NP][J_NP], dKr[J_NP][J_NP];
#pragma unroll
    for (int j = 0; j < J_NP; j++)
#pragma unroll
        for (int j1 = 0; j1 < J_NP; j1++) {
            dPc[j][j1] = B.dPcj_dS[(int64_t)(3 * j + j1) * nb + n];
            dKr[j][j1] = B.dKr_dS[(int64_t)(3 * j + j1) * nb + n];
        }
#pragma unroll
    for (int j = 0; j < J_NP; j++) {
        const uint32_t f = fl[j];
        if (!(f & F_EXU)) continue;
        const bool    mine = ((f & F_UPB) != 0) == (end == 0);  // upstream is this end
        const bool    both = (f & F_EXB) && (f & F_EXE);
        const double  dP = sm.q[j][Q_DP][lane], xi = sm.q[j][Q_XI][lane], mu = sm.q[j][Q_MU][lane];
        const double  y = sm.q[j][Q_Y][lane], muP = sm.q[j][Q_MUP][lane], tr = sm.q[j][Q_TR][lane];
        const double  xiP  = sm.q[j][Q_XIP][lane];
        const double  grho = M(-sm.q[j][Q_RHOP][lane], dGamma);
        const double  gown = M(-sm.q[j][end ? Q_RHOPE : Q_RHOPB][lane], dGamma);
        double tx[NR], a1[NR], a2[NR], dmu[NR], fk[NR];
        bool   safe = (f & F_SAFE) != 0;
#pragma unroll
        for (int i = 0; i < NR; i++) {
            const double xij = sm.x[j * NCOM + row0 + i][lane];
            tx[i] = M(M(xij, xi), tr);
            a1[i] = M(M(Akd, xij), xi);
            a2[i] = M(-tx[i], muP);
            safe  = safe && mid_range(tx[i]) && mid_range(a1[i]);
            p[i]  = end ? S(p[i], tx[i]) : A(p[i], tx[i]);
            if (both) p[i] = A(p[i], M(M(tx[i], gown), 0.5));
#pragma unroll
            for (int j1 = 0; j1 < J_NP; j1++) {
                const double t = M(tx[i], dPc[j][j1]);
                rs[j1][i]      = end ? S(rs[j1][i], t) : A(rs[j1][i], t);
            }
        }
        if (mine) {
            div_by(a2, mu, y, safe, dmu);
            div_by(a1, mu, y, safe, fk);
#pragma unroll
            for (int i = 0; i < NR; i++) {
                double tmp = M(M(M(sm.x[j * NCOM + row0 + i][lane], tr), xiP), dP);
                tmp        = A(tmp, M(dmu[i], dP));
                if (!both) tmp = A(tmp, M(tx[i], grho));
                p[i] = A(p[i], tmp);
#pragma unroll
                for (int j1 = 0; j1 < J_NP; j1++) rs[j1][i] = A(rs[j1][i], M(M(fk[i], dKr[j][j1]), dP));
            }
        }
    }
    // compact row k, column col: sec[(k NCOL + col) step]
    const double* sec  = CT::STAGED ? sm.sec + (size_t)end * CT::NENT * 32 + lane : B.dSec_dPri + n;
    const int64_t step = CT::STAGED ? 32 : nb;
    auto product = [&](const double (&r)[NR]) {
        double s[NCOL];
#pragma unroll
        for (int col = 0; col < NCOL; col++) {
            s[col] = *sec;
            sec += step;
        }
#pragma unroll
        for (int i = 0; i < NR; i++)
#pragma unroll
            for (int col = 0; col < NCOL; col++) acc[i][col] = A(acc[i][col], M(r[i], s[col]));
    };
#pragma unroll
    for (int j1 = 0; j1 < J_NP; j1++)
        if (fl[j1] & sd_me) product(rs[j1]);
    // the composition columns: those of phase j follow those of phase j - 1.
    // Entry (i, kk) of phase j at this end, or 0
    auto comp_load = [&](int j, int kk, double (&v)[3]) {
        const int64_t q = (int64_t)(j * NCOM + kk) * nb + n;
        v[0] = B.rhox[q], v[1] = B.xix[q], v[2] = B.mux[q];
    };
    auto comp_entry = [&](int j, uint32_t f, int kk, const double (&part)[3], double (&r)[NR]) {
        const bool    mine = ((f & F_UPB) != 0) == (end == 0);
        const bool    both = (f & F_EXB) && (f & F_EXE);
        const double  xi = sm.q[j][Q_XI][lane], tr = sm.q[j][Q_TR][lane];
        const double  rh = both ? M(part[0], 0.5) : part[0];
        double        tx[NR], v[NR];
        bool          safe = (f & F_SAFE) && mid_range(part[2]);
#pragma unroll
        for (int i = 0; i < NR; i++) {
            tx[i] = M(M(sm.x[j * NCOM + row0 + i][lane], xi), tr);
            safe  = safe && mid_range(tx[i]);
            v[i]  = M(M(-tx[i], rh), dGamma);
        }
        if (mine) {
            const double mu = sm.q[j][Q_MU][lane], y = sm.q[j][Q_Y][lane], dP = sm.q[j][Q_DP][lane];
            const double own = M(M(xi, tr), dP);
            double       num[NR], dmu[NR];
#pragma unroll
            for (int i = 0; i < NR; i++) num[i] = M(-tx[i], part[2]);
            div_by(num, mu, y, safe, dmu);
#pragma unroll
            for (int i = 0; i < NR; i++) {
                v[i] = A(v[i], M(M(M(sm.x[j * NCOM + row0 + i][lane], tr), part[1]), dP));
                v[i] = A(v[i], M(dmu[i], dP));
                r[i] = A(r[i], v[i]);
                if (row0 + i == kk) r[i] = A(r[i], own);
            }
        } else {
#pragma unroll
            for (int i = 0; i < NR; i++) r[i] = A(r[i], v[i]);
        }
    };
    if (!odd) {
#pragma unroll 1
        for (int j = 0; j < J_NP; j++) {
            const uint32_t f  = sm.f[j][lane];
            const int      nv = (f >> vsh) & 0xff;
            const bool     on = (f & F_EXU) && ((((f & F_UPB) != 0) == (end == 0)) || (f & ex_me));
            double         next[3] = {0, 0, 0};
            if (on && nv > 0) comp_load(j, 0, next);
#pragma unroll 1
            for (int kk = 0; kk < nv; kk++) {
                double       r[NR];
                const double part[3] = {next[0], next[1], next[2]};
#pragma unroll
                for (int i = 0; i < NR; i++) r[i] = 0;
                if (on) {
                    if (kk + 1 < nv) comp_load(j, kk + 1, next);
                    comp_entry(j, f, kk, part, r);
                }
                product(r);
            }
        }
    } else {
        // every column gathers what each phase's run of columns leaves in it
#pragma unroll 1
        for (int k = nsat; k < nsat + ncomp; k++) {
            double r[NR];
            int    j0 = nsat;
#pragma unroll
            for (int i = 0; i < NR; i++) r[i] = 0;
#pragma unroll 1
            for (int j = 0; j < J_NP; j++) {
                const uint32_t f    = sm.f[j][lane];
                const bool     mine = ((f & F_UPB) != 0) == (end == 0);
                const int      cnt  = (f >> (mine ? vsh : 24 - vsh)) & 0xff;
                if ((f & F_EXU) && (mine || (f & ex_me)) && k >= j0 && k < j0 + cnt) {
                    double part[3];
                    comp_load(j, k - j0, part);
                    comp_entry(j, f, k - j0, part, r);
                }
                j0 += (f >> vsh) & 0xff;
            }
            product(r);
        }
    }
#pragma unroll
    for (int i = 0; i < NR; i++) {
        if (row0 + i < first) continue;  // the group before has it
        double* d = dst + (int64_t)(row0 + i + 1) * NCOL * nc;
#pragma unroll
        for (int col = 0; col < NCOL; col++) {
            const double v = M(A(acc[i][col], col == 0 ? p[i] : 0.0), dt);
            *d             = end ? v : -v;
            d += nc;
        }
    }
}

template <int NCOM>
__global__ void __launch_bounds__(ConnTile<NCOM>::THREADS, ConnTile<NCOM>::MINB)
    k_conn_block(const __grid_constant__ ConnDev C, const __grid_constant__ ocpf_jac_bulk B, const int32_t* up,
                 const double* uprho, double dt, const __grid_constant__ ocpf_jac_out O)
{
    using CT = ConnTile<NCOM>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ConnStage<NCOM>* stage = reinterpret_cast<ConnStage<NCOM>*>(smem_raw);
    const int     tile = threadIdx.x / CT::TPT, w = (threadIdx.x % CT::TPT) >> 5, lane = threadIdx.x & 31;
    const int64_t c    = ((int64_t)blockIdx.x * CT::TILES + tile) * 32 + lane;
    const bool    live = c < C.nconn;
    const int     end = w & 1, g = w >> 1;
    if (live) {
        if (CT::STAGED) {
            // this end's rows; as many as the bulk has
            const int64_t nb = C.nb, n = end ? C.eId[c] : C.bId[c];
            int           rows = 0;
#pragma unroll
            for (int j = 0; j < J_NP; j++)
                rows += min((int)(B.pVnumCom[j * nb + n] & 0xff), NCOM) + (B.pSderExist[j * nb + n] ? 1 : 0);
            const int     cnt = min(rows, CT::NSEC) * CT::NCOL;
            double*       d   = stage[tile].sec + (size_t)end * CT::NENT * 32 + lane;
            const double* s   = B.dSec_dPri + n;
#pragma unroll 4
            for (int e = g; e < cnt; e += CT::G) copy8(d + e * 32, s + (int64_t)e * nb);
        }
        for (int j = w; j < J_NP; j += 2 * CT::G) stage_phase<NCOM>(C, B, up, uprho, c, j, lane, stage[tile]);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (!live) return;
    conn_rows<NCOM>(C, B, dt, O, c, lane, end, min(g * CT::NR, NCOM - CT::NR), g * CT::NR, stage[tile]);
}

template <int NCOM>
__global__ void __launch_bounds__(128) k_diag_rows(const ConnDev C, const ocpf_jac_bulk B, ocpf_jac_out O)
{
    constexpr int NCOL = NCOM + 1;
    const int64_t nb = C.nb, nc = C.nconn;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < NCOL * nb;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int     r = (int)(t / nb);
        const int64_t n = t - r * nb;
        double        d[NCOL];
        // accumulation block (src/OCPFluidMethod.cpp:1587-1596)
#pragma unroll
        for (int col = 0; col < NCOL; col++) d[col] = (r >= 1 && col == r) ? 1.0 : 0.0;
        if (r == 0) {
            d[0] = S(M(B.v[n], B.poroP[n]), B.vfP[n]);
#pragma unroll
            for (int k = 0; k < NCOM; k++) d[k + 1] = -B.vfi[(int64_t)k * nb + n];
        }
        for (int64_t q = C.adj_off[n]; q < C.adj_off[n + 1]; q++) {
            const int64_t a   = C.adj[q];
            const int64_t c   = a > 0 ? a - 1 : -a - 1;
            const double* src = a > 0 ? O.offEB : O.offBE;  // +bmatB = -offEB, -bmatE = -offBE
#pragma unroll
            for (int col = 0; col < NCOL; col++) d[col] = A(d[col], -src[(int64_t)(r * NCOL + col) * nc + c]);
        }
#pragma unroll
        for (int col = 0; col < NCOL; col++) O.diag[(int64_t)(r * NCOL + col) * nb + n] = d[col];
    }
}

template <int NCOM>
cudaError_t launch_jac(const ConnDev& C, const ocpf_jac_bulk& B, const int32_t* up, const double* uprho, double dt,
                       const ocpf_jac_out& O, int sms, cudaStream_t st)
{
    using CT = ConnTile<NCOM>;
    const int64_t t2 = (NCOM + 1) * C.nb;
    const int64_t g1 = (C.nconn + 32 * CT::TILES - 1) / (32 * CT::TILES);  // < 2^31: at most 2^30 connections
    const int     g2 = (int)std::min<int64_t>((t2 + 127) / 128, (int64_t)sms * 16);
    const int     smem = (int)sizeof(ConnStage<NCOM>) * CT::TILES;
    // per device; cheap, so on every launch
    cudaFuncSetAttribute(k_conn_block<NCOM>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (C.nconn > 0) k_conn_block<NCOM><<<(unsigned)g1, CT::THREADS, smem, st>>>(C, B, up, uprho, dt, O);
    if (C.nb > 0) k_diag_rows<NCOM><<<g2, 128, 0, st>>>(C, B, O);
    return cudaGetLastError();
}

}  // namespace
}  // namespace ocpf

struct ocpf_conn {
    int              device, sms;
    ocpf::ConnDev    d;
    void*            mem;
};

extern "C" int ocpf_conn_create(int64_t nbulk, int64_t nconn, const int64_t* bId, const int64_t* eId,
                                const double* area, int device, ocpf_conn** out)
{
    using namespace ocpf;
    if (!out) return OCPF_EINVAL;
    *out = nullptr;
    if (nbulk < 1 || nconn < 0 || (nconn > 0 && (!bId || !eId || !area))) return OCPF_EINVAL;
    if (nconn > 0x3fffffffLL) return OCPF_EINVAL;
    for (int64_t c = 0; c < nconn; c++)
        if (bId[c] < 0 || bId[c] >= nbulk || eId[c] < 0 || eId[c] >= nbulk || bId[c] == eId[c]) return OCPF_EINVAL;
    // per-bulk incident connections in connection order
    std::vector<int64_t> off(nbulk + 1, 0), adj(2 * nconn);
    for (int64_t c = 0; c < nconn; c++) {
        off[bId[c] + 1]++;
        off[eId[c] + 1]++;
    }
    for (int64_t n = 0; n < nbulk; n++) off[n + 1] += off[n];
    std::vector<int64_t> pos(off.begin(), off.end() - 1);
    for (int64_t c = 0; c < nconn; c++) {
        adj[pos[bId[c]]++] = c + 1;
        adj[pos[eId[c]]++] = -(c + 1);
    }
    int prev = 0;
    cudaGetDevice(&prev);
    if (cudaSetDevice(device) != cudaSuccess) return OCPF_ECUDA;
    ocpf_conn* h = new (std::nothrow) ocpf_conn;
    int        rc = h ? OCPF_OK : OCPF_ENOMEM;
    if (rc == OCPF_OK) {
        std::memset(h, 0, sizeof(*h));
        h->device = device;
        cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, device);
        const size_t b1 = sizeof(int64_t) * (size_t)nconn, b2 = sizeof(double) * (size_t)nconn;
        const size_t b3 = sizeof(int64_t) * (size_t)(nbulk + 1), b4 = sizeof(int64_t) * (size_t)(2 * nconn);
        const size_t tot = 2 * b1 + b2 + b3 + b4 + 5 * 256;
        if (cudaMalloc(&h->mem, tot) != cudaSuccess) {
            rc = OCPF_ENOMEM;
        } else {
            char* p    = (char*)h->mem;
            auto  take = [&p](size_t b) {
                char* q = p;
                p += (b + 255) / 256 * 256;
                return q;
            };
            int64_t* dB  = (int64_t*)take(b1);
            int64_t* dE  = (int64_t*)take(b1);
            double*  dA  = (double*)take(b2);
            int64_t* dO  = (int64_t*)take(b3);
            int64_t* dJ  = (int64_t*)take(b4);
            cudaError_t e = cudaSuccess;
            if (nconn > 0) {
                e = cudaMemcpy(dB, bId, b1, cudaMemcpyHostToDevice);
                if (e == cudaSuccess) e = cudaMemcpy(dE, eId, b1, cudaMemcpyHostToDevice);
                if (e == cudaSuccess) e = cudaMemcpy(dA, area, b2, cudaMemcpyHostToDevice);
                if (e == cudaSuccess) e = cudaMemcpy(dJ, adj.data(), b4, cudaMemcpyHostToDevice);
            }
            if (e == cudaSuccess) e = cudaMemcpy(dO, off.data(), b3, cudaMemcpyHostToDevice);
            if (e != cudaSuccess) rc = OCPF_ECUDA;
            h->d = ConnDev{nbulk, nconn, dB, dE, dA, dO, dJ};
        }
    }
    if (rc != OCPF_OK && h) {
        if (h->mem) cudaFree(h->mem);
        delete h;
        h = nullptr;
    }
    if (prev != device) cudaSetDevice(prev);
    *out = h;
    return rc;
}

extern "C" int ocpf_conn_destroy(ocpf_conn* h)
{
    if (!h) return OCPF_OK;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(h->device);
    cudaFree(h->mem);
    if (prev != h->device) cudaSetDevice(prev);
    delete h;
    return OCPF_OK;
}

extern "C" int ocpf_fim_upwind(ocpf_conn* h, const ocpf_jac_bulk* bk, int32_t* upblock, double* upblock_rho,
                               void* stream)
{
    using namespace ocpf;
    if (!h || !bk || !upblock || !upblock_rho || !bk->phaseExist || !bk->S || !bk->rho || !bk->Pj || !bk->depth)
        return OCPF_EINVAL;
    if (h->d.nconn == 0) return OCPF_OK;
    int prev = 0;
    cudaGetDevice(&prev);
    if (prev != h->device) cudaSetDevice(h->device);
    const int64_t t = J_NP * h->d.nconn;
    const int     g = (int)std::min<int64_t>((t + 255) / 256, (int64_t)h->sms * 8);
    k_upwind<<<g, 256, 0, (cudaStream_t)stream>>>(h->d, *bk, upblock, upblock_rho);
    const cudaError_t e = cudaGetLastError();
    if (prev != h->device) cudaSetDevice(prev);
    return e == cudaSuccess ? OCPF_OK : OCPF_ECUDA;
}

extern "C" int ocpf_fim_jacobian(ocpf_conn* h, int nc, double dt, const ocpf_jac_bulk* bk, const int32_t* upblock,
                                 const double* upblock_rho, ocpf_jac_out* out, void* stream)
{
    using namespace ocpf;
    if (!h || !bk || !out || !out->diag || !out->offEB || !out->offBE) return OCPF_EINVAL;
    if (h->d.nconn > 0 && (!upblock || !upblock_rho)) return OCPF_EINVAL;
    const ocpf_jac_bulk& B = *bk;
    if (!B.phaseExist || !B.pSderExist || !B.pVnumCom || !B.xi || !B.mu || !B.muP || !B.xiP || !B.rhoP || !B.xij ||
        !B.rhox || !B.xix || !B.mux || !B.dSec_dPri || !B.vfP || !B.vfi || !B.kr || !B.Pj || !B.dKr_dS ||
        !B.dPcj_dS || !B.v || !B.poroP || !B.depth)
        return OCPF_EINVAL;
    int prev = 0;
    cudaGetDevice(&prev);
    if (prev != h->device) cudaSetDevice(h->device);
    cudaError_t  e  = cudaSuccess;
    cudaStream_t st = (cudaStream_t)stream;
    switch (nc) {
        case 3: e = launch_jac<4>(h->d, B, upblock, upblock_rho, dt, *out, h->sms, st); break;
        case 6: e = launch_jac<7>(h->d, B, upblock, upblock_rho, dt, *out, h->sms, st); break;
        case 9: e = launch_jac<10>(h->d, B, upblock, upblock_rho, dt, *out, h->sms, st); break;
        case 12: e = launch_jac<13>(h->d, B, upblock, upblock_rho, dt, *out, h->sms, st); break;
        default:
            if (prev != h->device) cudaSetDevice(prev);
            return OCPF_EUNSUPPORTED;
    }
    if (prev != h->device) cudaSetDevice(prev);
    return e == cudaSuccess ? OCPF_OK : OCPF_ECUDA;
}

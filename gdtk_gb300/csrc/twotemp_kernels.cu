// twotemp_kernels.cu -- the multi-temperature thermochemical reactor for a two-temperature gas, eight
// lanes per cell, compiled with FMA contraction, with the rate constants and equilibrium constants in
// log form (one exp where the reference takes pows and an exp), the NASA-9 curves in polynomial form and exp, ln
// and divisions on the integer pipe: results differ from the reference's evaluation order in rounding
// only (tested to 1e-8 in Y, 1e-7 relative in T, T_ve and p).
//
// kinetics/multi_temperature_thermochemical_reactor.d:137-294 (opCall) and :334-431 (Cash-Karp RKF
// on the concentrations and u_ve), with
//   * rate constants once per subcycle at the clamped T (reaction_mechanism.d:49-63): Gibbs energies
//     at p = P_atm and T_ve = T (:204-218, two_temperature_gas.d:469-482), forward Arrhenius or Park
//     (rate_constant.d:72-75, 364-393: T_eff = T^s T_ve^(1-s)) or (modified) Marrone-Treanor over either
//     (rate_constant.d:395-566), backward k_f(T, T_ve = T) / K_c(T)
//     (reaction.d:94-143, 26-52);
//   * tick rates and q - L (reaction.d:290-311, 416-440; reaction_mechanism.d:74-96);
//   * energy exchange (energy_exchange_system.d:93-104): Landau-Teller (energy_exchange_mechanism.d:
//     83-101) with Millikan-White / Park high-temperature relaxation times (relaxation_time.d:27-175),
//     evaluated once per subcycle on the subcycle's gas state, and Marrone-Treanor coupling with
//     impartial, Marrone-Treanor or modified Marrone-Treanor dissociation (energy_exchange_mechanism.d:
//     228-241, exchange_chemistry_coupling.d:41-227; G_appear and G_vanish on the subcycle's state) on
//     the current stage's tick rates;
//   * T from u by direct inversion and T_ve by Newton iteration (two_temperature_gas.d:95-117, 656-700).
// A cell that fails keeps its input state and gets the reference's failure as its status.
#include <cuda_runtime.h>

#include <cmath>

#include "cea_thermo.h"
#include "chem_types.h"
#define GDTK_FN static __device__ __noinline__   // one copy each: fetching inlined ones costs more than the calls
#include "fast_exp.h"
#include "cea_poly.cuh"
#include "twotemp.h"

namespace gdtk {
namespace {

constexpr double R_universal = 8.31451;       // gas/physical_constants.d:13
constexpr double P_atm = 101.325e3;           // gas/physical_constants.d:16
constexpr double Avogadro = 6.02214e23;       // gas/physical_constants.d:19
constexpr double T_REF = 298.15;              // two_temperature_gas.d:26
constexpr double SMALL_MOLE_FRACTION = 1.0e-15;   // gas_model.d:42
constexpr double IGAMMA_SWITCH = 1.0e-7;      // exchange_chemistry_coupling.d:24
constexpr double IGAMMA_OVERFLOW = 0.001;     // exchange_chemistry_coupling.d:25
constexpr double H_MIN = 1.0e-15;             // multi_temperature_thermochemical_reactor.d:31
constexpr double R_INV = 1.0 / R_universal;
constexpr double LN_PATM_R = 0x1.2d0f0af013269p+3;   // ln(P_atm / R_universal) = 9.408086270233257
constexpr double ALLOWABLE_MASSF_ERROR = 1.0e-3;
constexpr int MAX_EEM = 64;

// exp on the integer pipe (fast_exp.h).  The update kernel stages its table in shared memory once per block.
__device__ const uint64_t kExp2Table[GDTK_EXP2_TABLE_SIZE] = GDTK_EXP2_TABLE_INIT;
__shared__ uint64_t s_exp2[GDTK_EXP2_TABLE_SIZE];
__device__ __forceinline__ double ex(double x) { return gdtk_exp(x, s_exp2); }

// NASA-9 Cp, h and s of cea_thermo_curves.d:55-137 (cea_thermo.h's segment choice and blending,
// cea_coeffs) in Horner form with the reciprocal temperature rT = 1 / T: the reference's divisions by T,
// T^2 and the small integers become multiplications.
__device__ double cea_h_r(const MechView& m, int isp, double T, double rT, double logT, int& err) {
    const double* s = m.sp(isp);
    if (T < s[SP_TLOW]) return s[SP_HLOW] - s[SP_CPLOW] * (s[SP_TLOW] - T);
    if (T > s[SP_THIGH]) return s[SP_HHIGH] + s[SP_CPHIGH] * (T - s[SP_THIGH]);
    double a[9];
    if (!cea_coeffs(m, isp, T, a)) { err = CELL_CEA_RANGE; return 0.0; }
    // h/R = -a0/T + a1 ln T + a2 T + a3 T^2/2 + a4 T^3/3 + a5 T^4/4 + a6 T^5/5 + a7
    const double poly = fma(T, fma(T, fma(T, a[6] * 0.2, a[5] * 0.25), a[4] * (1.0 / 3.0)), a[3] * 0.5);
    const double h = fma(-a[0], rT, fma(a[1], logT, a[7])) + T * fma(T, poly, a[2]);
    return s[SP_R] * h;
}
struct Gas2T {
    MechView m;
    const Species2T* sp;
    int electron;
    __device__ double R(int i) const { return m.sp(i)[SP_R]; }
    // two_temperature_gas.d:427-445, 538-545, 558-590
    // rTve = 1 / T_ve, logTve = ln T_ve
    __device__ double e_ve(int i, double Tve, double rTve, double logTve, int& err) const {
        if (i == electron) return 1.5 * R(i) * Tve;
        return cea_h_r(m, i, Tve, rTve, logTve, err) - sp[i].cp_tr * (Tve - T_REF) - sp[i].h_f;
    }
    __device__ double e_tr(int i, double T) const {
        if (i == electron) return 0.0;
        return sp[i].cp_tr * (T - T_REF) + sp[i].h_f - R(i) * T;
    }
    __device__ double e_ve_mix(const double* Y, double Tve, int& err) const {
        const double r = 1.0 / Tve, lt = log(Tve);
        double e = 0.0;
        for (int i = 0; i < m.nsp; ++i) e += Y[i] * e_ve(i, Tve, r, lt, err);
        return e;
    }
    __device__ double e_tr_mix(const double* Y, double T) const {
        double e = 0.0;
        for (int i = 0; i < m.nsp; ++i)
            if (i != electron) e += Y[i] * e_tr(i, T);
        return e;
    }
};

// An Arrhenius (at T) or Park (at T_e = T^s T_ve^(1-s)) rate constant from the record's A, n, C, s, in log
// form: A exp(n ln T_e - C / T_e) with ln T_e = s ln T + (1 - s) ln T_ve from the logs of the subcycle
// (rate_constant.d:72-75, 364-393 evaluate the same expression with three pow calls and an exp).
// Temperatures enter as reciprocals (rT = 1 / T), formed once per subcycle where the reference divides.
__device__ double base_rc(int model, const double* d, double rT, double lnT, double lnTve) {
    if (model == RATE_PARK) {
        const double lnTe = d[RD_S] * lnT + (1.0 - d[RD_S]) * lnTve;
        return d[0] * ex(d[1] * lnTe - d[2] * ex(-lnTe));
    }
    return d[0] * ex(d[1] * lnT - d[2] * rT);
}

// rate_constant.d:397-404 at the temperature whose reciprocal is rT
__device__ __forceinline__ double Q_mt(double rT, double D, double theta) {
    const double num = 1 - ex(-D * rT);
    const double den = 1 - ex(-theta * rT);
    return gdtk_div(num, den);
}

// Forward rate constant of reaction ir at (T, T_ve): Arrhenius, Park, or the (modified) Marrone-Treanor
// non-equilibrium factor times the underlying one (rate_constant.d:438-447, 541-554).
__device__ double forward_rc(const int* r, const double* d, double rT, double rTve, double lnT, double lnTve) {
    const int model = r[RX_FRC];
    if (model != RATE_MT && model != RATE_MMT) return base_rc(model, d, rT, lnT, lnTve);
    const double kEQ = base_rc(r[RX_BASE], d, rT, lnT, lnTve);
    const double TD = d[RD_MT_TD], th = d[RD_MT_THETA];
    if (model == RATE_MT) {
        const double rU = gdtk_rcp(d[RD_MT_U]);
        const double rGamma = rTve - rT - rU;   // 1 / Gamma
        const double Q_T = Q_mt(rT, TD, th), Q_Gamma = Q_mt(rGamma, TD, th), Q_Tv = Q_mt(rTve, TD, th),
                     Q_U = Q_mt(-rU, TD, th);
        return gdtk_div(kEQ * Q_T * Q_Gamma, Q_Tv * Q_U);
    }
    const double Uinv = d[RD_MT_U] * rT + gdtk_rcp(d[RD_MT_USTAR]);
    const double rTF = rTve - rT - Uinv;   // 1 / T_F
    const double Q_T = Q_mt(rT, TD, th), Q_TF = Q_mt(rTF, TD, th), Q_Tv = Q_mt(rTve, TD, th),
                 Q_U = Q_mt(-Uinv, TD, th);
    return gdtk_div(d[RD_MT_NB] * kEQ * Q_T * Q_TF, Q_Tv * Q_U);
}

// Knab's equation (39) and its small-iG and overflow forms (exchange_chemistry_coupling.d:41-69).
__device__ double L_knab(double iG, double D, double Th) {
    if (fabs(iG) < IGAMMA_SWITCH)
        return 0.5 * (D - Th * R_universal) + iG * (Th * Th * R_universal * R_universal - D * D) * (R_INV / 12.0);
    if (iG > IGAMMA_OVERFLOW)
        return gdtk_div(R_universal * Th, ex(Th * iG) - 1.0) - D * ex(-D * R_INV * iG);
    return gdtk_div(R_universal * Th, ex(Th * iG) - 1.0) - gdtk_div(D, ex(D * R_INV * iG) - 1.0);
}

// Energy brought in (ga) and removed (gv) per dissociation at (T, T_ve), J/mol
// (exchange_chemistry_coupling.d:94-126 impartial, 152-174 Marrone-Treanor, 204-220 modified).
// rT = 1 / T, rTv = 1 / T_v
__device__ void coupling(const Eem2T& e, double rT, double rTv, double& ga, double& gv) {
    const double th = e.Thetav;
    if (e.coupling == CPL_IMPARTIAL) {
        ga = 0.5 * (e.D - th * R_universal);
        gv = L_knab(rTv - rT, e.D, th);   // (T - T_v) / (T T_v)
    } else if (e.coupling == CPL_MARRONE_TREANOR) {
        const double rU = gdtk_rcp(e.U);
        gv = L_knab(rTv - rT - rU, e.D, th);
        ga = gdtk_div(R_universal * th, ex(-th * rU) - 1.) - gdtk_div(e.D, ex(-e.D * R_INV * rU) - 1.);
    } else {
        const double TD = e.D;
        const double Uinv = e.aU * rT + gdtk_rcp(e.Ustar);
        const double T_F_inv = rTv - rT - Uinv;
        gv = R_universal * (gdtk_div(th, ex(th * T_F_inv) - 1.) - gdtk_div(TD, ex(TD * T_F_inv) - 1.)) + e.nb * R_universal * TD;
        ga = R_universal * (gdtk_div(th, ex(-th * Uinv) - 1.) - gdtk_div(TD, ex(-TD * Uinv) - 1.));
    }
}

// ---------------------------------------------------------------- the update
// Eight lanes per cell in a persistent grid, four cells to a warp: species, reactions and exchange mechanisms are
// spread over the lanes, and a cell's vectors lie in its slice of shared memory.  One thread per cell issued about
// 5,900 FP64 instructions per attempt and warp (32 cells), most of them over tables that every lane walked for
// itself, with 13 of 32 lanes active and a warp waiting for its longest cell; eight lanes issue about 930 for
// 4 cells, a cell's attempt takes a fifth of the time, and cells are handed out as groups come free.
// 65,536 non-equilibrium air cells over 2e-7 s: 181 -> 64 ms; one cell 14.4 -> 3.0 ms.  FP64 issue (69% busy at
// 16,384 cells) and instruction fetch bound it.
// All groups of a warp stay in step: every sync and shuffle is over the whole warp, in loops uniform over it.
// The operations per cell are those of the subcycle and attempt loops of
// multi_temperature_thermochemical_reactor.d:137-294.
constexpr int GL = 8;
constexpr unsigned FULL = 0xffffffffu;
constexpr int UPDATE_BLOCK = 256;   // 3 blocks per SM: 65.3 ms where 2 take 67.8 and 1 81.6, and 4 (64 registers) 64.4

// Cash-Karp stage coefficients (multi_temperature_thermochemical_reactor.d:334-431)
__constant__ double CK_A[5][5] = {
    {1. / 5., 0, 0, 0, 0},
    {3. / 40., 9. / 40., 0, 0, 0},
    {3. / 10., -9. / 10., 6. / 5., 0, 0},
    {-11. / 54., 5. / 2., -70. / 27., 35. / 27., 0},
    {1631. / 55296., 175. / 512., 575. / 13824., 44275. / 110592., 253. / 4096.}};

using gdtk_fast::abs_bits;
using gdtk_fast::ge_pos;
using gdtk_fast::gt_pos;
using gdtk_fast::larger_abs;
using gdtk_fast::lt_pos;

// offsets of a cell's vectors in its slice, in doubles
struct Layout2T {
    int y0, yT, K, wf, wb, net, kf, kb, G, Y, de, xa, xb, ga, gv, total;
    __host__ __device__ Layout2T(int nsp, int nr, int ncpl) {
        const int nv = nsp + 1;
        y0 = 0; yT = nv; K = 2 * nv; wf = 8 * nv; wb = wf + nr; net = wb + nr; kf = net + nr; kb = kf + nr; G = kb + nr;
        Y = G + nsp; de = Y + nsp; xa = de + nsp; xb = xa + nsp; ga = xb + nsp; gv = ga + ncpl;
        total = (gv + ncpl) | 1;
    }
};

// sum over a group's lanes, in every lane
__device__ __forceinline__ double group_sum(double v) {
    v += __shfl_xor_sync(FULL, v, 1);
    v += __shfl_xor_sync(FULL, v, 2);
    v += __shfl_xor_sync(FULL, v, 4);
    return v;
}

// BIG: with coefficients beyond the reaction table's 126, which are read from the mechanism (the test for them costs 2.7%).
template <bool BIG>
__global__ void __launch_bounds__(UPDATE_BLOCK, 3) two_temperature_update_kernel(const TwoTArgs a) {
    extern __shared__ double smem[];
    MechView m;
    m.bind(a.mech_i, a.mech_d);
    const int nsp = m.nsp, nr = m.nr, nv = nsp + 1, ncpl = a.ncpl;
    // tables: thermo, efficiencies, tick rates, per-species stoichiometry
    double* TH = smem;
    double* EFF = TH + nsp * GDTK_TH_STRIDE;
    const int n_eff = a.neff * nsp;
    int* IT = reinterpret_cast<int*>(EFF + n_eff);
    for (int k = threadIdx.x; k < GDTK_EXP2_TABLE_SIZE; k += blockDim.x) s_exp2[k] = kExp2Table[k];
    for (int k = threadIdx.x; k < nsp * GDTK_TH_STRIDE; k += blockDim.x) TH[k] = a.thermo[k];
    for (int k = threadIdx.x; k < n_eff; k += blockDim.x) EFF[k] = a.eff[k];
    for (int k = threadIdx.x; k < a.n_tab; k += blockDim.x) IT[k] = a.tab[k];
    __syncthreads();
    const int* RX = IT;                       // per reaction: reactants, products (8 bits each), their coefficients, set
    const int* ST = IT + 5 * nr;              // first entry of each species (nsp + 1)
    const int* SE = ST + nsp + 1;             // entries: reaction, high word of nu
    const Layout2T lay(nsp, nr, ncpl);
    const int lane = threadIdx.x & 31, gl = lane & (GL - 1), leader0 = lane & ~(GL - 1);
    double* S = EFF + n_eff + (a.n_tab + 1) / 2 + (size_t)(threadIdx.x / GL) * lay.total;
    double *y0 = S + lay.y0, *yT = S + lay.yT, *K = S + lay.K, *wf = S + lay.wf, *wb = S + lay.wb, *net = S + lay.net,
           *kf = S + lay.kf, *kb = S + lay.kb, *G = S + lay.G, *Y = S + lay.Y, *de = S + lay.de, *xa = S + lay.xa,
           *xb = S + lay.xb, *gas = S + lay.ga, *gvs = S + lay.gv;
    const Species2T* sp = a.species;
    const int electron = a.electron;
    const double tI = a.t_interval, rnv = 1.0 / nv, T_lower = m.T_lower(), T_upper = m.T_upper();
    auto R = [&](int i) { return m.sp(i)[SP_R]; };
    // two_temperature_gas.d:427-445, 538-545, 558-590: vibration-electronic energy and heat capacity of a species
    auto ve = [&](int i, double Tv, double rTv, double lnTv, double& e, double& cv, int& err) {
        if (i == electron) { e = 1.5 * R(i) * Tv; cv = 1.5 * R(i); return; }
        double H, Cp;
        gdtk_fast::sp_H_Cp(TH, i, Tv, lnTv, rTv, rTv * rTv, H, Cp, err);
        e = fma(R(i), H, -fma(sp[i].cp_tr, Tv - T_REF, sp[i].h_f));
        cv = fma(R(i), Cp, -sp[i].cp_tr);
    };
    unsigned long long my_steps = 0;
    int c = 0, phase = 0, cycle = 0, attempt = 0, fail = 0, err = 0;
    bool have = false, exhausted = false;
    double rho = 0.0, rrho = 0.0, T = 0.0, Tve = 0.0, p = 0.0, t = 0.0, h = 0.0, dt_suggest = 0.0, dtSave = 0.0;
    double u_total = 0.0, u = 0.0, u_ve = 0.0, LT = 0.0;
    // Tick rates at y (net w_f - w_b beside them), then dy/dt into out: species, and the energy exchange in out[nsp]
    // (reaction_mechanism.d:82-95; the Landau-Teller sum LT holds for the subcycle)
    auto rates = [&](bool act, const double* y, double* out, bool energy) {
        if (act) {
            for (int r = gl; r < nr; r += GL) {
                const int *x = RX + 5 * r, set = x[4];
                double f = kf[r], b = kb[r];
                if (set >= 0) {
                    const double* ef = EFF + set * nsp;
                    double mc = 0.0;
                    for (int i = 0; i < nsp; ++i) mc = fma(ef[i], y[i], mc);
                    f *= mc;
                    b *= mc;
                }
                for (int k = 0; k < (x[2] & 7); ++k) {
                    const double v = y[(x[0] >> (8 * k)) & 255];
                    int n = (x[2] >> (3 + 7 * k)) & 127;
                    if (BIG && n == 127) n = m.rx(r)[RX_REAC_COEFF + k];
                    for (; n > 0; --n) f *= v;
                }
                for (int k = 0; k < (x[3] & 7); ++k) {
                    const double v = y[(x[1] >> (8 * k)) & 255];
                    int n = (x[3] >> (3 + 7 * k)) & 127;
                    if (BIG && n == 127) n = m.rx(r)[RX_PROD_COEFF + k];
                    for (; n > 0; --n) b *= v;
                }
                wf[r] = f;
                wb[r] = b;
                net[r] = f - b;
            }
        }
        __syncwarp(FULL);
        if (out) {
            double rate = 0.0;
            if (act) {
                for (int i = gl; i < nsp; i += GL) {
                    double v = 0.0;
                    for (int k = ST[i]; k < ST[i + 1]; ++k) v = fma(__hiloint2double(SE[2 * k + 1], 0), net[SE[2 * k]], v);
                    out[i] = v;
                }
                if (energy)
                    for (int k = gl; k < ncpl; k += GL) {
                        const Coupling2T cp = a.cpl[k];   // nu of the dissociating species in the coupled reaction
                        const double f = wf[cp.reaction], b = wb[cp.reaction];
                        const bool up = __double_as_longlong(cp.nu) > 0;   // prod = nu f, loss = nu b; or -nu b, -nu f
                        const double pr = up ? f : b, lo = up ? b : f;
                        rate = fma(pr, gas[k], fma(-lo, gvs[k], rate));
                    }
            }
            rate = group_sum(rate);
            if (act && gl == 0) out[nsp] = fma(rate, rrho, LT);
            __syncwarp(FULL);
        }
    };
    while (true) {
        if (!exhausted) {   // refill: at most one atomic per warp
            const unsigned need = __ballot_sync(FULL, !have && gl == 0);
            if (need) {
                unsigned base = 0;
                if (lane == 0) base = atomicAdd(a.counter, (unsigned)__popc(need));
                base = __shfl_sync(FULL, base, 0);
                const unsigned pos = base + __popc(need & ((1u << leader0) - 1u));
                if (!have && pos < (unsigned)a.ncell) {
                    c = (int)pos;
                    have = true;
                    phase = 0;
                }
                exhausted = base + __popc(need) >= (unsigned)a.ncell;
            }
        }
        if (!__any_sync(FULL, have)) {
            if (exhausted) break;
            continue;
        }
        bool act = have;
        if (__any_sync(FULL, have && phase == 0)) {   // a cell's state
            const bool start = have && phase == 0;
            double e_ve = 0.0, e_tr = 0.0;
            if (start) {
                rho = a.rho[c];
                T = a.T[c]; Tve = a.Tve[c]; p = a.p[c];
                fail = 0; err = 0;
                dt_suggest = a.dt_chem[c]; dtSave = dt_suggest; u = 0.0; u_ve = 0.0; t = 0.0; cycle = 0;
                if (isnan(rho) || rho <= 0.0) {
                    fail = CELL_BAD_INPUT;
                } else {
                    rrho = gdtk_rcp(rho);
                    const double lt = gdtk_log(Tve), rt = gdtk_rcp(Tve);
                    for (int i = gl; i < nsp; i += GL) {
                        const double y = a.massf[(size_t)i * a.ncell + c];
                        Y[i] = y;
                        const double v = y * rho * (R(i) * R_INV);   // 1 / M_i = R_i / R_universal
                        y0[i] = v < 1.0e-30 ? 0.0 : v;   // gas_model.d:237-256
                        double e, cv;
                        ve(i, Tve, rt, lt, e, cv, err);
                        e_ve += y * e;
                        if (i != electron) e_tr += y * (sp[i].cp_tr * (T - T_REF) + sp[i].h_f - R(i) * T);
                    }
                    if (a.max_subcycles <= 0) fail = CELL_MAX_SUBCYCLES;
                }
            }
            e_ve = group_sum(e_ve);
            e_tr = group_sum(e_tr);
            if (start) {
                u_total = e_tr + e_ve;
                if (gl == 0) y0[nsp] = e_ve;
            }
            __syncwarp(FULL);
        }
        act = have && !fail;
        const bool setup = act && phase <= 1;
        if (__any_sync(FULL, setup)) {   // a subcycle's rate constants, relaxation times and exchange terms
            double logT = 0.0, logTve = 0.0, rT = 0.0, rTve = 0.0, T13 = 0.0, sqrtT = 0.0;
            if (setup) {
                logT = gdtk_log(T); logTve = gdtk_log(Tve);
                rT = gdtk_rcp(T); rTve = gdtk_rcp(Tve);
                T13 = ex(logT * (-1. / 3.));
                sqrtT = ex(0.5 * logT);
                // reaction.d:94-143 (multi-temperature branch) at the clamped T: G / RT at (T, T_ve = T, p = P_atm)
                double Tc = T, lTc = logT, rTc = rT;
                if (lt_pos(Tc, T_lower)) { Tc = T_lower; lTc = gdtk_log(Tc); rTc = gdtk_rcp(Tc); }
                if (gt_pos(Tc, T_upper)) { Tc = T_upper; lTc = gdtk_log(Tc); rTc = gdtk_rcp(Tc); }
                for (int i = gl; i < nsp; i += GL)
                    G[i] = gdtk_fast::sp_G(TH, i, Tc, lTc, rTc, rTc * rTc, lTc + 1.0, 1.0 - lTc, err);
            }
            __syncwarp(FULL);
            double mol = 0.0;
            if (setup) {
                double lTc = logT, rTc = rT;
                if (lt_pos(T, T_lower)) { lTc = gdtk_log(T_lower); rTc = gdtk_rcp(T_lower); }
                if (gt_pos(T, T_upper)) { lTc = gdtk_log(T_upper); rTc = gdtk_rcp(T_upper); }
                for (int r = gl; r < nr; r += GL) {
                    const int* x = m.rx(r);
                    const double* d = m.rxd(r);
                    double lnKc = 0.0;
                    if (x[RX_FRC] == RATE_FROM_EQ || x[RX_BRC] == RATE_FROM_EQ) {   // reaction.d:26-52
                        double dG = 0.0;
                        int nuSum = 0;
                        for (int k = 0; k < x[RX_NPART]; ++k) {
                            const int nu = x[RX_PART_NU + k];
                            const double g = G[x[RX_PART + k]];
                            dG = nu == 1 ? dG + g : nu == -1 ? dG - g : fma((double)nu, g, dG);
                            nuSum += nu;
                        }
                        lnKc = nuSum == 0 ? -dG : nuSum == 1 ? (LN_PATM_R - lTc) - dG
                                                             : fma((double)nuSum, LN_PATM_R - lTc, -dG);   // K_p (P_atm / R T)^sum(nu)
                    }
                    if (x[RX_FRC] != RATE_FROM_EQ) {
                        kf[r] = forward_rc(x, d, rTc, rTve, lTc, logTve);
                        kb[r] = (x[RX_BRC] == RATE_FROM_EQ) ? forward_rc(x, d, rTc, rTc, lTc, lTc) * ex(-lnKc)
                                                            : d[3] * ex(d[4] * lTc - d[5] * rTc);
                    } else {
                        const double b = d[3] * ex(d[4] * lTc - d[5] * rTc);
                        kb[r] = b;
                        kf[r] = b * ex(lnKc);   // the backward rate constant at the state itself (reaction.d:131)
                    }
                }
                for (int i = gl; i < nsp; i += GL) mol += Y[i] * (R(i) * R_INV);
            }
            mol = group_sum(mol);
            double md = 1.0e6;
            const bool est = setup && phase == 0 && !(dt_suggest > tI) && dt_suggest <= 0.0;
            if (__any_sync(FULL, est)) {   // the first step, reaction_mechanism.d:161-203
                __syncwarp(FULL);
                rates(est, y0, nullptr, false);
                if (est)
                    for (int i = gl; i < nsp; i += GL) {
                        double q = 0.0, L = 0.0;
                        for (int k = ST[i]; k < ST[i + 1]; ++k) {
                            const double nu = __hiloint2double(SE[2 * k + 1], 0);
                            const int r = SE[2 * k];
                            q += nu > 0.0 ? nu * wf[r] : -nu * wb[r];
                            L += nu > 0.0 ? nu * wb[r] : -nu * wf[r];
                        }
                        if (y0[i] > 0.0 && fabs(q - L) > 1.0e-30) {
                            const double dt = (q > 10000.0 * L) ? gdtk_div(y0[i], L + 1.0e-50) : fabs(gdtk_div(y0[i], q - L));
                            md = fmin(md, dt);
                        }
                    }
                for (int x = 1; x < GL; x <<= 1) md = fmin(md, __shfl_xor_sync(FULL, md, x));
            }
            if (setup && phase == 0) {
                h = dt_suggest > tI ? tI : dt_suggest <= 0.0 ? fmax(fmin(1.0e-3 * md, 1.0e-10), 1.0e-15) : dt_suggest;
                phase = 1;
            }
            if (setup) {   // mole fractions, number densities, Y (e_ve(T) - e_ve(T_ve))
                const double rmol = gdtk_rcp(mol);
                for (int i = gl; i < nsp; i += GL) {
                    const double n_i = Y[i] * (R(i) * R_INV);
                    xa[i] = n_i * rmol;
                    xb[i] = Avogadro * rho * n_i;
                    double e1 = 0.0, e2 = 0.0, cv;
                    if ((a.relaxing >> i) & 1u) {
                        ve(i, T, rT, logT, e1, cv, err);
                        ve(i, Tve, rTve, logTve, e2, cv, err);
                    }
                    de[i] = Y[i] * (e1 - e2);
                }
            }
            __syncwarp(FULL);
            double lt = 0.0;
            if (setup) {
                const double patm = p * (1.0 / P_atm);
                const double htc2 = sqrtT * (50e3 * rT) * (50e3 * rT);
                for (int k = gl; k < a.neem; k += GL) {
                    const Eem2T& e = a.eem[k];
                    if (e.kind == EEM_LANDAU_TELLER) {   // relaxation_time.d:27-175; a rare collider has none
                        if (gt_pos(xa[e.q], SMALL_MOLE_FRACTION)) {
                            double tau = gdtk_div(ex(fma(e.a, T13, -e.b)), xa[e.q] * patm);   // the partial pressure in atm
                            if (e.rt != RT_MILLIKAN_WHITE) tau += gdtk_rcp(e.sigma * xb[e.q] * (e.rt == RT_PARK_HTC ? sqrtT : htc2));
                            // a negative time or none (at T <= 0) relaxes nothing
                            if ((unsigned long long)__double_as_longlong(tau) <= 0x7ff0000000000000ull) lt += gdtk_div(de[e.p], tau);
                        }
                    } else {
                        double g0, g1;
                        coupling(e, rT, rTve, g0, g1);
                        const double nu = fabs(a.cpl[e.slot].nu);
                        gas[e.slot] = nu * g0;
                        gvs[e.slot] = nu * g1;
                    }
                }
            }
            LT = setup ? 0.0 : LT;
            lt = group_sum(lt);
            for (int x = 1; x < GL; x <<= 1) err |= __shfl_xor_sync(FULL, err, x);
            if (setup) {
                LT = lt;
                dtSave = dt_suggest;
                h = fmin(h, tI - t);
                attempt = 0;
                phase = 2;
                if (a.max_attempts <= 0) fail = CELL_MAX_ATTEMPTS;
            }
            __syncwarp(FULL);
        }
        act = have && !fail;
        bool done = false;
        if (__any_sync(FULL, act)) {   // one Cash-Karp attempt
#pragma unroll 1
            for (int s = 0; s < 6; ++s) {
                double* Ks = K + s * nv;
                rates(act, s == 0 ? y0 : yT, Ks, true);
                if (act && s < 5)
                    for (int i = gl; i < nv; i += GL) {
                        double v = CK_A[s][0] * K[i];
                        for (int j = 1; j <= s; ++j) v = fma(CK_A[s][j], K[j * nv + i], v);
                        yT[i] = fma(h, v, y0[i]);
                    }
                __syncwarp(FULL);
            }
            double e2 = 0.0, tot = 0.0;
            if (act)
                for (int i = gl; i < nv; i += GL) {
                    const double b51 = 37. / 378., b53 = 250. / 621., b54 = 125. / 594., b56 = 512. / 1771.,
                                 b41 = 2825. / 27648., b43 = 18575. / 48384., b44 = 13525. / 55296., b45 = 277. / 14336.,
                                 b46 = 1.0 / 4.0;
                    const double k1 = K[i], k3 = K[2 * nv + i], k4 = K[3 * nv + i], k5 = K[4 * nv + i], k6 = K[5 * nv + i], y = y0[i];
                    const double o = fma(h, fma(b56, k6, fma(b54, k4, fma(b53, k3, b51 * k1))), y);
                    const double o4 = fma(h, fma(b46, k6, fma(b45, k5, fma(b44, k4, fma(b43, k3, b41 * k1)))), y);
                    const double e = gdtk_div(o - o4, fma(a.tol, larger_abs(y, o), a.tol));
                    yT[i] = o;
                    e2 = fma(e, e, e2);
                    if (i < nsp) {   // conc2massf (gas_model.d:258-271)
                        const double v = o * m.sp(i)[SP_M] * rrho;
                        const double yi = lt_pos(v, 1.0e-30) ? 0.0 : v;
                        Y[i] = yi;
                        tot += yi;
                    }
                }
            e2 = group_sum(e2);
            tot = group_sum(tot);
            bool ok = false;
            if (act) {
                const double en2 = e2 * rnv;   // the square of the error norm: en^-0.2 = en2^-0.1
                ok = en2 <= 1.0;
                double scale = 10.0;
                if (en2 != 0.0) {
                    scale = fmax(0.9 * ex(-0.1 * gdtk_log(en2)), 0.2);
                    if (ok) scale = fmin(scale, 10.0);
                }
                dt_suggest = scale * h;
                if (gl == 0) ++my_steps;
                if (ok && gt_pos(abs_bits(tot - 1.0), ALLOWABLE_MASSF_ERROR)) ok = false;
                if (ok) {   // the attempt ends the subcycle
                    t += h;
                    for (int i = gl; i < nv; i += GL) y0[i] = yT[i];
                    if (dt_suggest > h) h = fmin(dt_suggest, h * (1.0 + 10.0 / 100.0));
                } else {
                    h = gdtk_div(h, 10.0);
                    if (h < H_MIN) fail = CELL_H_MIN;
                    else if (++attempt == a.max_attempts) fail = CELL_MAX_ATTEMPTS;
                }
            }
            __syncwarp(FULL);
            if (__any_sync(FULL, ok)) {   // updateFromRhoU (two_temperature_gas.d:95-117, 656-700): T directly, T_ve by Newton
                double sA = 0.0, sB = 0.0;
                if (ok)
                    for (int i = gl; i < nsp; i += GL)
                        if (i != electron) {
                            sA = fma(Y[i], fma(sp[i].cp_tr, T_REF, -sp[i].h_f), sA);
                            sB = fma(Y[i], sp[i].cp_tr - R(i), sB);
                        }
                sA = group_sum(sA);
                sB = group_sum(sB);
                double Tg = Tve, lg = 0.0, rg = 0.0, dT = 0.0;
                if (ok) {
                    u_ve = y0[nsp];
                    u = u_total - u_ve;
                    T = gdtk_div(u + sA, sB);
                    lg = gdtk_log(Tg);
                    rg = gdtk_rcp(Tg);
                }
                bool on = ok, failed = false;
                int e = 0;
                // 40 iterations, |dT| < 1e-9 K, or the guess itself when its energy is within 1e-5 J/kg
#pragma unroll 1
                for (int it = 0; it <= 40; ++it) {
                    if (!__any_sync(FULL, on)) break;
                    double f = 0.0, cv = 0.0;
                    if (on)
                        for (int i = gl; i < nsp; i += GL) {
                            double ei, ci;
                            ve(i, Tg, rg, lg, ei, ci, e);
                            f = fma(Y[i], ei, f);
                            cv = fma(Y[i], ci, cv);
                        }
                    f = group_sum(f);
                    cv = group_sum(cv);
                    if (on) {
                        f -= u_ve;
                        if (it == 0 && lt_pos(abs_bits(f), 1e-5)) {
                            on = false;
                        } else if (it == 40) {
                            on = false;
                            failed = gt_pos(abs_bits(dT), 1e-3);
                        } else {
                            dT = -gdtk_div(f, cv);
                            const double x = dT * rg;
                            Tg += dT;
                            if (lt_pos(abs_bits(dT), 1.0e-9)) on = false;
                            else {
                                lg = gdtk_fast::ln_step(lg, x, Tg);
                                rg = gdtk_rcp(Tg);
                            }
                        }
                    }
                }
                for (int x = 1; x < GL; x <<= 1) e |= __shfl_xor_sync(FULL, e, x);
                double pr = 0.0;
                if (ok) {
                    if (e) failed = true;
                    if (!failed) Tve = Tg;
                    for (int i = gl; i < nsp; i += GL) pr = fma(rho * Y[i] * R(i), i == electron ? Tve : T, pr);
                }
                pr = group_sum(pr);
                if (ok) {
                    if (failed) {
                        fail = CELL_NEWTON_FAIL;
                    } else {
                        p = pr;
                        if (ge_pos(t, tI)) {
                            if (cycle == 0) dtSave = dt_suggest;
                            done = true;
                        } else if (++cycle == a.max_subcycles) {
                            fail = CELL_MAX_SUBCYCLES;
                        } else {
                            phase = 1;
                        }
                    }
                }
            }
        }
        if (done && err) { fail = CELL_CEA_RANGE; done = false; }
        double tot = 0.0;
        if (__any_sync(FULL, done)) {
            if (done)
                for (int i = gl; i < nsp; i += GL) tot += Y[i];
            tot = group_sum(tot);
        }
        if (have && fail) {
            if (a.status && gl == 0) a.status[c] = fail;
            have = false;
        } else if (done) {
            const double rtot = gdtk_rcp(tot);
            for (int i = gl; i < nsp; i += GL) a.massf[(size_t)i * a.ncell + c] = Y[i] * rtot;
            if (gl == 0) {
                a.T[c] = T;
                a.Tve[c] = Tve;
                a.p[c] = p;
                if (a.u) a.u[c] = u;
                if (a.u_ve) a.u_ve[c] = u_ve;
                a.dt_chem[c] = dtSave;
                if (a.status) a.status[c] = CELL_OK;
            }
            have = false;
        }
        __syncwarp(FULL);
    }
    if (a.steps && my_steps) atomicAdd(a.steps, my_steps);
}

__global__ void two_temperature_thermo_pT_kernel(const Thermo2TArgs a) {
    Gas2T g;
    g.m.bind(a.mech_i, a.mech_d);
    g.sp = a.species;
    g.electron = a.electron;
    const int nsp = g.m.nsp;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < a.ncell; c += gridDim.x * blockDim.x) {
        double Y[GDTK_MAX_SPECIES];
        for (int i = 0; i < nsp; ++i) Y[i] = a.massf[(size_t)i * a.ncell + c];
        const double T = a.T[c], Tve = a.Tve[c];
        double denom = 0.0;   // two_temperature_gas.d updateDensity
        for (int i = 0; i < nsp; ++i) denom += Y[i] * g.R(i) * (i == g.electron ? Tve : T);
        int err = 0;
        a.rho[c] = a.p[c] / denom;
        a.u[c] = g.e_tr_mix(Y, T);
        a.u_ve[c] = g.e_ve_mix(Y, Tve, err);
    }
}

int grid_for_cells(int n, int block, int sm_count) {
    long long g = ((long long)n + block - 1) / block;
    const long long cap = (long long)sm_count * 16;
    if (g > cap) g = cap;
    return g < 1 ? 1 : (int)g;
}

}  // namespace

cudaError_t launch_two_temperature_update(const TwoTArgs& a, int nsp, int nr, int sm_count, cudaStream_t s) {
    if (a.ncell <= 0) return cudaSuccess;
    if (a.neem > MAX_EEM || !a.counter) return cudaErrorInvalidValue;
    // as many blocks per SM as are resident (three of 256 threads), each with as many warps (four cells each) as fit, or
    // as a share of the batch needs
    constexpr size_t LIMIT = 227 * 1024 - 2 * GDTK_EXP2_TABLE_SIZE * 8;
    const size_t tables = (size_t)(nsp * GDTK_TH_STRIDE + a.neff * nsp + (a.n_tab + 1) / 2) * 8;
    const size_t per_warp = (size_t)Layout2T(nsp, nr, a.ncpl).total * (32 / GL) * 8;
    const auto kernel = a.big ? two_temperature_update_kernel<true> : two_temperature_update_kernel<false>;
    cudaError_t e = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LIMIT);
    if (e != cudaSuccess) return e;
    if (tables + per_warp > LIMIT) return cudaErrorInvalidConfiguration;
    const long long warps = ((long long)a.ncell + 32 / GL - 1) / (32 / GL);
    int per_block = UPDATE_BLOCK / 32;
    while (per_block > 1 && tables + per_warp * per_block > LIMIT) --per_block;
    const long long fair = (warps + sm_count - 1) / sm_count;
    if (fair < per_block) per_block = (int)fair;
    const size_t smem = tables + per_warp * per_block;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)kernel, 32 * per_block, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    long long grid = (long long)sm_count * per_sm;
    const long long want = (warps + per_block - 1) / per_block;
    if (grid > want) grid = want;
    e = cudaMemsetAsync(a.counter, 0, sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    kernel<<<(unsigned)grid, 32 * per_block, smem, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_two_temperature_thermo_pT(const Thermo2TArgs& a, int sm_count, cudaStream_t s) {
    if (a.ncell <= 0) return cudaSuccess;
    two_temperature_thermo_pT_kernel<<<grid_for_cells(a.ncell, 128, sm_count), 128, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace gdtk

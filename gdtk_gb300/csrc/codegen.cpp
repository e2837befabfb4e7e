// codegen.cpp -- writes the mechanism as CUDA, compiles it with NVRTC for the device at hand, and
// launches it.
//
// The generated part is small: compile-time sizes and tolerances, the species constants, and
// two functions -- gen_kc (rate constants: a loop over a __constant__ table of the Arrhenius
// reactions, the pressure-dependent ones straight-line) and gen_rhs (production/loss rates,
// straight-line) -- in which every species index, stoichiometric coefficient, third-body
// efficiency and Arrhenius parameter is a literal or a table entry.  The integrator around them is chem_fast.cuh.  The reference
// interprets its reaction objects at run time (kinetics/reaction_mechanism.d:82-96,
// reaction.d:145-149, 267-311, 394-456); its legacy GPU path generated source in a similar
// spirit, from prep-chem's compact notation (eilmer/utils/prep-cuda-gpu-chem-kernel.py).
#include "codegen.h"

#include <cuda.h>
#include <nvrtc.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <sstream>
#include <stdexcept>
#include <tuple>
#include <sys/stat.h>
#include <unistd.h>

#include "cea_thermo.h"
#include "chem_types.h"
#include "fast_exp.h"
#include "chem_launch.h"

namespace gdtk {

extern const char* const kFastCuhSource;
extern const char* const kFastExpSource;
extern const char* const kCeaPolySource;
extern const char* const kGroupCuhSource;

namespace {

constexpr double R_universal = 8.31451;
constexpr int kGroupBlock = 512;   // most threads of a block of the kernel with a group of lanes per cell

std::string lit(double v) {   // exact double literal
    char buf[64];
    std::snprintf(buf, sizeof buf, "%a", v);
    std::string s(buf);
    if (v == 0.0) return "0.0";
    return s;
}

// ---- driver entry points, resolved through the runtime (no link-time libcuda dependency)
struct Driver {
    CUresult (*moduleLoadData)(CUmodule*, const void*) = nullptr;
    CUresult (*moduleUnload)(CUmodule) = nullptr;
    CUresult (*moduleGetFunction)(CUfunction*, CUmodule, const char*) = nullptr;
    CUresult (*funcSetAttribute)(CUfunction, CUfunction_attribute, int) = nullptr;
    CUresult (*launchKernel)(CUfunction, unsigned, unsigned, unsigned, unsigned, unsigned, unsigned, unsigned,
                             CUstream, void**, void**) = nullptr;
    CUresult (*occupancy)(int*, CUfunction, int, size_t) = nullptr;
    CUresult (*getErrorString)(CUresult, const char**) = nullptr;
};

template <typename F>
void resolve(const char* name, F& fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t e = cudaGetDriverEntryPointByVersion(name, &p, 12000, cudaEnableDefault, &q);
    if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !p)
        throw std::runtime_error(std::string("cannot resolve driver entry point ") + name);
    fn = reinterpret_cast<F>(p);
}

Driver& driver() {
    static Driver d;
    static std::once_flag once;
    static std::string failure;
    std::call_once(once, [] {
        try {
            resolve("cuModuleLoadData", d.moduleLoadData);
            resolve("cuModuleUnload", d.moduleUnload);
            resolve("cuModuleGetFunction", d.moduleGetFunction);
            resolve("cuFuncSetAttribute", d.funcSetAttribute);
            resolve("cuLaunchKernel", d.launchKernel);
            resolve("cuOccupancyMaxActiveBlocksPerMultiprocessor", d.occupancy);
            resolve("cuGetErrorString", d.getErrorString);
        } catch (std::exception& e) {
            failure = e.what();
        }
    });
    if (!failure.empty()) throw std::runtime_error(failure);
    return d;
}

void cu_check(CUresult r, const char* what) {
    if (r == CUDA_SUCCESS) return;
    const char* s = "unknown";
    if (driver().getErrorString) driver().getErrorString(r, &s);
    throw std::runtime_error(std::string(what) + ": " + s);
}

// Integer power of a symbol, in the order of D's std.math pow(x, int) (binary exponentiation).
std::string ipow_expr(const std::string& x, int n) {
    if (n == 1) return x;
    if (n == 2) return "(" + x + " * " + x + ")";
    std::string p, v = x;
    unsigned m = (unsigned)n;
    bool have = false;
    while (true) {
        if (m & 1u) { p = have ? "(" + p + " * " + v + ")" : v; have = true; }
        m >>= 1;
        if (!m) break;
        v = "(" + v + " * " + v + ")";
    }
    return p;
}

struct Part { int isp; int nu; };

std::vector<Part> participants(const ReactionHost& r) {
    std::vector<int> sp;
    for (auto& x : r.reac) sp.push_back(x.first);
    for (auto& x : r.prod) sp.push_back(x.first);
    std::sort(sp.begin(), sp.end());
    sp.erase(std::unique(sp.begin(), sp.end()), sp.end());
    std::vector<Part> out;
    for (int isp : sp) {
        int nu1 = 0, nu2 = 0;
        for (auto& x : r.reac) if (x.first == isp) { nu1 = x.second; break; }
        for (auto& x : r.prod) if (x.first == isp) { nu2 = x.second; break; }
        out.push_back({isp, nu2 - nu1});
    }
    return out;
}

// ln k = ln A + n ln T - C / T as an expression; empty if A == 0.
std::string log_arrhenius(const RateConstHost& rc) {
    if (rc.model == RATE_ARRHENIUS2) {   // ln k = logA + B T - C/T (rate_constant.d:112-115)
        std::string e = lit(rc.A);
        if (rc.n != 0.0) e = "fma(" + lit(rc.n) + ", T, " + e + ")";
        if (rc.C != 0.0) e = "fma(" + lit(-rc.C) + ", rT, " + e + ")";
        return e;
    }
    if (rc.A <= 0.0) return "";
    std::string e = lit(std::log(rc.A));
    if (rc.n != 0.0) e = "fma(" + lit(rc.n) + ", lnT, " + e + ")";
    if (rc.C != 0.0) e = "fma(" + lit(-rc.C) + ", rT, " + e + ")";
    return e;
}

// k = A T^n as products when C == 0 and n is a small integer (no exponential needed).
bool power_arrhenius(const RateConstHost& rc, std::string& out) {
    if (rc.model != RATE_ARRHENIUS || rc.C != 0.0 || rc.n != std::floor(rc.n) || std::fabs(rc.n) > 4) return false;
    int n = (int)rc.n;
    if (n == 0) { out = lit(rc.A); return true; }
    out = lit(rc.A) + " * " + ipow_expr(n > 0 ? "T" : "rT", n > 0 ? n : -n);
    return true;
}

// k = A T^n exp(-C/T) as an expression (products, one exponential, or 0).
std::string arrhenius_expr(double A, double n, double C) {
    RateConstHost rc;
    rc.A = A; rc.n = n; rc.C = C;
    std::string e;
    if (power_arrhenius(rc, e)) return e;
    e = log_arrhenius(rc);
    return e.empty() ? std::string("0.0") : "gdtk_exp(" + e + ", etab)";
}

// Rate constants of the pressure-dependent reactions (rate_constant.d:155-160, 258-287, 338-350), from the
// third-body concentration Mc, as one function over a table: log10 and pow(10, x) are written as
// ln x / ln 10 and exp(x ln 10), and k_b = k_f / K_c.
const char* const kFalloffSource = R"(
struct FallRec { double lnA, n, mC, A, lnA0, n0, mC0, A0, lfc, a, x1, x2, x3; int model, flags, pw, pw0, np, nusum, idx, pad;
                 int sp[8]; double nu[8]; };
__device__ __forceinline__ double fall_arrhenius(double lnA, double n, double mC, double A, int pw, double T, double lnT, double rT,
                                                 const uint64_t* etab) {
  if (pw == 98) return 0.0;
  if (pw == 99) return gdtk_exp(fma(mC, rT, fma(n, lnT, lnA)), etab);
  const double b = pw > 0 ? T : rT;
  double k = A;
  for (int m = 0; m < abs(pw); ++m) k *= b;
  return k;
}
__device__ __noinline__ void falloff_rates(const FallRec& R, double T, double lnT, double rT, double Mc, const double* g, int gs,
                                           const uint64_t* etab, double& kf, double& kb) {
  const double INV_LN10 = 0x1.bcb7b1526e50ep-2, LN10 = 0x1.26bb1bbb55516p+1;
  const double kinf = fall_arrhenius(R.lnA, R.n, R.mC, R.A, R.pw, T, lnT, rT, etab);
  const double k0 = fall_arrhenius(R.lnA0, R.n0, R.mC0, R.A0, R.pw0, T, lnT, rT, etab);
  if (R.model == 4) {   // Yungster-Rabinowitz
    const double pr = gdtk_div(k0 * Mc, kinf), lpr = gdtk_log(pr);
    const double fc = fma(R.a, gdtk_exp(R.x1 * rT, etab), (1.0 - R.a) * gdtk_exp(R.x2 * rT, etab));
    kf = gdtk_div(__dmul_rn(kinf * gdtk_div(pr, 1.0 + pr), fc), fma(lpr, lpr, 1.0));
  } else {
    kf = gdtk_div(k0 * kinf * Mc, fma(k0, Mc, kinf));
    if (R.model == 3) {   // Troe
      const double lpr = gdtk_log(fmax(gdtk_div(k0 * Mc, kinf), 1.0e-30)) * INV_LN10;
      double lfc = R.lfc;
      if (!(R.flags & 1)) {
        double fcent = (1.0 - R.a) * gdtk_exp(R.x3 * T, etab);
        if (R.flags & 2) fcent = fma(R.a, gdtk_exp(R.x1 * T, etab), fcent);
        if (R.flags & 4) fcent += gdtk_exp(R.x2 * rT, etab);
        lfc = gdtk_log(fmax(fcent, 1.0e-30)) * INV_LN10;
      }
      const double numer = lpr + fma(-0.67, lfc, -0.4);
      const double frac = gdtk_div(numer, fma(-0.14, numer, fma(-1.27, lfc, 0.75)));
      kf *= gdtk_exp(gdtk_div(lfc, fma(frac, frac, 1.0)) * LN10, etab);
    }
  }
  double dg = 0.0;
  for (int k = 0; k < R.np; ++k) dg = fma(R.nu[k], g[R.sp[k] * gs], dg);
  kb = kf * gdtk_exp(-fma((double)R.nusum, GDTK_LN_PATM_R - lnT, -dg), etab);
}
)";

// A row of GDTK_FALL_TAB.
std::string falloff_record(const ReactionHost& r, int ir) {
    const RateConstHost& f = r.frc;
    auto power = [](double A, double n, double C) {
        if (C == 0.0 && n == std::floor(n) && std::fabs(n) <= 4) return (int)n;
        return A <= 0.0 ? 98 : 99;
    };
    auto ln = [](double A) { return A > 0.0 ? std::log(A) : 0.0; };
    const bool troe = f.model == RATE_TROE, given = f.troe_flags & TROE_FCENT;
    // -1 / x for exp(-T / x), which is 0 for x = 0: finite, so that it is a literal
    auto inv = [](double x) { return std::max(-1.0e300, std::min(1.0e300, -1.0 / x)); };
    std::ostringstream o, sp, nu;
    int np = 0, nusum = 0;
    for (auto& pp : participants(r)) {
        if (pp.nu == 0) continue;
        sp << (np ? ", " : "") << pp.isp;
        nu << (np ? ", " : "") << lit((double)pp.nu);
        nusum += pp.nu;
        ++np;
    }
    if (np == 0) { sp << "0"; nu << "0.0"; }
    o << "  {" << lit(ln(f.A)) << ", " << lit(f.n) << ", " << lit(-f.C) << ", " << lit(f.A) << ", " << lit(ln(f.A0)) << ", "
      << lit(f.n0) << ", " << lit(-f.C0) << ", " << lit(f.A0) << ", "
      << lit(troe && given ? std::log10(std::max(f.Fcent, 1.0e-30)) : 0.0) << ", " << lit(f.a) << ", "
      << lit(troe ? inv(f.T1) : -f.T1) << ", " << lit(-f.T2) << ", " << lit(troe ? inv(f.T3) : 0.0) << ", "
      << (f.model == RATE_LH ? 2 : troe ? 3 : 4) << ", " << f.troe_flags << ", " << power(f.A, f.n, f.C) << ", "
      << power(f.A0, f.n0, f.C0) << ", " << np << ", " << nusum << ", " << ir << ", 0, {" << sp.str() << "}, {" << nu.str()
      << "}},\n";
    return o.str();
}

}  // namespace

FastKernel::~FastKernel() {
    if (module) driver().moduleUnload((CUmodule)module);
    if (d_thermo) cudaFree(d_thermo);
    if (d_exp) cudaFree(d_exp);
}

std::vector<double> fast_thermo_table(const GasModelHost& gm) {
    const int nsp = gm.n_species();
    PackedMech pm = pack(gm, nullptr);   // reference-form curve ends (cea_thermo_curves.d:46-53)
    MechView v;
    v.bind(pm.I.data(), pm.D.data());
    std::vector<double> t((size_t)nsp * 120, 0.0);
    for (int i = 0; i < nsp; ++i) {
        const CeaCurveHost& c = gm.curves[i];
        const double* s = v.sp(i);
        const double R = R_universal / gm.M[i];
        double* th = t.data() + (size_t)i * 120;
        th[0] = s[SP_TLOW];
        th[1] = s[SP_THIGH];
        th[2] = s[SP_HLOW] / R;
        th[3] = s[SP_HHIGH] / R;
        th[4] = s[SP_CPLOW] / R;
        th[5] = s[SP_CPHIGH] / R;
        th[6] = s[SP_SLOW] / R;
        th[7] = s[SP_SHIGH] / R;
        th[8] = std::log(s[SP_TLOW]);
        th[9] = std::log(s[SP_THIGH]);
        // segment count as integer bits; per break k = 1..nseg-1 the blend window [lo, hi] of
        // cea_thermo_curves.d:150-182 (break -/+ blend/2, the reference's arithmetic) and 1 / blend
        const int64_t nseg_bits = c.nseg;
        std::memcpy(&th[10], &nseg_bits, sizeof nseg_bits);
        for (int k = 1; k < c.nseg; ++k) {
            th[10 + k] = c.breaks[k] - 0.5 * c.blends[k - 1];
            th[13 + k] = c.breaks[k] + 0.5 * c.blends[k - 1];
            th[16 + k] = 1. / c.blends[k - 1];
            if (!(th[10 + k] > 0.0)) throw NoFastKernel("thermo curve blend window below 0 K");
        }
        for (int sg = 0; sg < c.nseg; ++sg) {
            const double* a = c.coeffs.data() + 9 * sg;
            double* h = th + 24 + 24 * sg;
            // H/R = -a0/T + a1 lnT + a7 + T (a2 + T (a3/2 + T (a4/3 + T (a5/4 + T a6/5))))
            h[0] = -a[0]; h[1] = a[1]; h[2] = a[2]; h[3] = a[3] / 2.0; h[4] = a[4] / 3.0; h[5] = a[5] / 4.0;
            h[6] = a[6] / 5.0; h[7] = a[7];
            // Cp/R = a0/T^2 + a1/T + a2 + T (a3 + T (a4 + T (a5 + T a6)))
            for (int k = 0; k < 7; ++k) h[8 + k] = a[k];
            // G/RT = H/RT - S/R
            h[15] = -a[0] / 2.0; h[16] = a[1]; h[17] = a[7]; h[18] = a[2]; h[19] = -a[8];
            h[20] = -a[3] / 2.0; h[21] = -a[4] / 6.0; h[22] = -a[5] / 12.0; h[23] = -a[6] / 20.0;
        }
    }
    return t;
}

// The temperature range where every species takes the same curve segment and blend of
// cea_thermo_curves.d:150-182 (so that the mixture's H/R is one polynomial there): species curves
// with at least two segments and the same break and blend between the first two, from the highest lower end to the
// lowest upper end or blend with a third segment.
// Unroll factors of the rate-constant loops (reaction table, species G/RT): two independent
// iterations in flight give the FP64 pipe work while one waits on its table loads.
int env_int(const char* name, int dflt) {
    const char* e = std::getenv(name);
    return (e && *e) ? std::max(1, std::atoi(e)) : dflt;
}
int kc_unroll() { return env_int("GDTK_KC_UNROLL", 1); }
int g_unroll() { return env_int("GDTK_G_UNROLL", 1); }
// Reactions between compiler fences in gen_rhs (0: none); the fences bound how far the scheduler
// hoists the k_f, k_b loads, and with them the registers held.
int rhs_fence() {
    const char* e = std::getenv("GDTK_RHS_FENCE");
    return (e && *e) ? std::max(0, std::atoi(e)) : 4;
}

// A third-body sum over the species (leaf: the efficiency, 0 where absent) as chem_group.cuh's third_body_sum: pairs with the
// second product fused, then the zero-padded pairwise tree of chem_fast.cuh's sum_pairwise.
std::string third_body_sum(const std::vector<double>& leaf, int lo, int n) {
    auto c = [](int i) { return "c[" + std::to_string(i) + "]"; };
    auto product = [&](int i) { return leaf[i] == 0.0 ? std::string() : leaf[i] == 1.0 ? c(i) : "__dmul_rn(" + lit(leaf[i]) + ", " + c(i) + ")"; };
    if (n == 1) return product(lo);
    if (n == 2 && lo + 1 < (int)leaf.size() && leaf[lo] != 0.0 && leaf[lo + 1] != 0.0 && leaf[lo + 1] != 1.0)
        return "fma(" + lit(leaf[lo + 1]) + ", " + c(lo + 1) + ", " + product(lo) + ")";
    const std::string a = third_body_sum(leaf, lo, n / 2);
    std::string b;
    if (lo + n / 2 < (int)leaf.size()) b = third_body_sum(leaf, lo + n / 2, n / 2);
    if (a.empty() || b.empty()) return a.empty() ? b : a;
    return "(" + a + " + " + b + ")";
}

// Whether the kernel with a group of lanes per cell (chem_group.cuh) takes the mechanism: every reaction in
// its tables, and no code form asked for that only the one-thread-per-cell kernel has.
bool group_kernel_takes(const MechanismHost& mh, size_t n_table, size_t n_falloff) {
    for (const char* e : {"GDTK_KC_UNROLLED", "GDTK_KB_EXP", "GDTK_PHASE_CLOCKS"}) {
        const char* v = std::getenv(e);
        if (v && v[0] == '1') return false;
    }
    if (n_table + n_falloff != mh.reactions.size()) return false;
    for (auto& r : mh.reactions)
        for (auto* side : {&r.reac, &r.prod}) {
            if (side->size() > 4) return false;
            for (auto& x : *side) if (x.second < 1 || x.second > 7) return false;
        }
    return true;
}

bool mix_thermo_range(const GasModelHost& gm, double& tlo, double& thi) {
    const int nsp = gm.n_species();
    if (nsp == 0) return false;
    PackedMech pm = pack(gm, nullptr);
    MechView v;
    v.bind(pm.I.data(), pm.D.data());
    const CeaCurveHost& c0 = gm.curves[0];
    tlo = -1e300;
    thi = 1e300;
    for (int i = 0; i < nsp; ++i) {
        const CeaCurveHost& c = gm.curves[i];
        if (c.nseg < 2 || c0.nseg < 2 || c.breaks[1] != c0.breaks[1] || c.blends[0] != c0.blends[0]) return false;
        tlo = std::max(tlo, v.sp(i)[SP_TLOW]);
        thi = std::min(thi, v.sp(i)[SP_THIGH]);
        if (c.nseg > 2) thi = std::min(thi, c.breaks[2] - 0.5 * c.blends[1]);
    }
    return thi > tlo;
}

// Largest |G_i / R T| of each species over [tlo, thi] (log-spaced samples plus the curve breaks),
// from the same NASA-9 curves, blends and extrapolation the kernels use.
std::vector<double> species_g_bound(const GasModelHost& gm, double tlo, double thi) {
    const int nsp = gm.n_species();
    PackedMech pm = pack(gm, nullptr);
    MechView v;
    v.bind(pm.I.data(), pm.D.data());
    std::vector<double> Ts;
    const int n = 4000;
    for (int k = 0; k <= n; ++k) Ts.push_back(tlo * std::pow(thi / tlo, (double)k / n));
    for (auto& c : gm.curves)
        for (double b : c.breaks)
            if (b > tlo && b < thi) { Ts.push_back(b); Ts.push_back(b * (1 - 1e-9)); Ts.push_back(b * (1 + 1e-9)); }
    std::vector<double> out(nsp, 0.0);
    for (int i = 0; i < nsp; ++i) {
        const double Ri = R_universal / gm.M[i];
        for (double T : Ts) {
            int err = 0;
            const double lT = std::log(T);
            const double g = (cea_h(v, i, T, lT, err) - T * cea_s(v, i, T, lT, err)) / (Ri * T);
            out[i] = (err || !std::isfinite(g)) ? 1e300 : std::max(out[i], std::fabs(g));
        }
    }
    return out;
}

// Reactions whose k_b = k_f / K_c is formed as k_f (R T / P_atm)^(sum nu) prod_i E_i^nu_i with
// E_i = exp(G_i / R T) formed once per species (GDTK_KB_EXP=1 keeps one exp per reaction).  Only where
// every partial product stays inside exp(+-600) over the mechanism's temperature limits, so that no
// product can overflow or underflow.
std::vector<bool> kb_product_reactions(const GasModelHost& gm, const MechanismHost& mh) {
    std::vector<bool> out(mh.reactions.size(), false);
    const char* e = std::getenv("GDTK_KB_EXP");
    if (e && e[0] == '1') return out;
    const std::vector<double> gb = species_g_bound(gm, mh.T_lower, mh.T_upper);
    const double lcf = std::max(std::fabs(std::log(mh.T_lower * R_universal / 101325.0)),
                                std::fabs(std::log(mh.T_upper * R_universal / 101325.0)));
    for (size_t ir = 0; ir < mh.reactions.size(); ++ir) {
        const ReactionHost& r = mh.reactions[ir];
        if (r.frc.pressure_dependent() || r.frc.model != RATE_ARRHENIUS || r.brc.model != RATE_FROM_EQ) continue;
        double bound = 0.0;
        int nusum = 0, np = 0;
        for (auto& pp : participants(r)) {
            bound += std::abs(pp.nu) * gb[pp.isp];
            nusum += pp.nu;
            np += pp.nu != 0;
        }
        bound += std::abs(nusum) * lcf;
        out[ir] = np <= 8 && bound <= 600.0;
    }
    return out;
}

bool any_kb_products(const GasModelHost& gm, const MechanismHost& mh) {
    for (bool b : kb_product_reactions(gm, mh)) if (b) return true;
    return false;
}

// Per-thread method vector (doubles): the ODE method's stage storage, and room for the
// species' Y_i R_i plus two sets of 12 mixture coefficients during T(rho, u).
int fast_vec_doubles(const GasModelHost& gm, const MechanismHost& mh) {
    const int nsp = gm.n_species();
    int vec = (mh.method == METHOD_RKF ? 6 : 3) * nsp;
    double tlo, thi;
    if (mix_thermo_range(gm, tlo, thi)) vec = std::max(vec, nsp + 24);
    int nfall = 0;   // third-body concentrations of pressure-dependent rates, beside G/RT
    for (auto& r : mh.reactions) nfall += r.frc.pressure_dependent() ? 1 : 0;
    // G/RT, the falloff concentrations, then E_i and 1/E_i for the product-form k_b
    return std::max(vec, (any_kb_products(gm, mh) ? 3 * nsp : nsp) + nfall);
}

// The tables of chem_group.cuh: rate-constant records, tick-rate records (both sorted so that the lanes of a
// round take the same path), and the q and L sums as tasks, dealt whole to 4, 8, 16 or 32 lanes, longest first.
std::string group_tables(const GasModelHost& gm, const MechanismHost& mh, const std::vector<int>& table_rx,
                         const std::vector<bool>& kbp, const std::vector<std::vector<std::pair<int, double>>>& sets,
                         const std::vector<int>& set_of, GroupShape& shape) {
    const int nsp = gm.n_species(), nr = (int)mh.reactions.size();
    std::ostringstream o;
    auto high = [](double v) {
        uint64_t b;
        std::memcpy(&b, &v, 8);
        return (unsigned)(b >> 32);
    };
    int nfall = 0;
    for (auto& r : mh.reactions) nfall += r.frc.pressure_dependent() ? 1 : 0;
    bool any = false;
    for (int ir : table_rx) any = any || kbp[ir];
    o << "#define GDTK_ANY_KBP " << (any ? 1 : 0) << "\n#define GDTK_NKC " << table_rx.size() << "\n#define GDTK_NSETS "
      << sets.size() << "\n#define GDTK_GRP_BLOCK " << kGroupBlock << "\n";
    // GRP_CELL of chem_group.cuh (checked there)
    const int nsets = (int)sets.size();
    shape.cell_doubles = (4 * nsp + 2 * nr + std::max(2 * nr, std::max(3 * nsp + nfall, nsp + 24)) + nsets +
                          (mh.method == METHOD_RKF ? 6 : 3) * nsp) | 1;
    // rate constants, by path
    struct Kc { int ir, mode, pw, np, nusum; std::vector<Part> parts; };
    std::vector<Kc> kc;
    for (int ir : table_rx) {
        const ReactionHost& r = mh.reactions[ir];
        Kc k{ir, 0, 99, 0, 0, {}};
        for (auto& pp : participants(r))
            if (pp.nu) { k.parts.push_back(pp); k.nusum += pp.nu; }
        k.np = (int)k.parts.size();
        k.mode = r.frc.model == RATE_ARRHENIUS ? (r.brc.model == RATE_FROM_EQ ? 0 : 1) : 2;
        if (k.mode == 0 && kbp[ir]) k.mode = 3;
        std::string e;
        if (power_arrhenius(r.frc, e)) k.pw = (int)r.frc.n;
        kc.push_back(k);
    }
    auto kc_key = [](const Kc& k) { return std::make_tuple(k.mode, k.mode == 3 && k.pw != 99, k.np, std::abs(k.nusum)); };
    std::stable_sort(kc.begin(), kc.end(), [&](const Kc& a, const Kc& b) { return kc_key(a) < kc_key(b); });
    o << "struct GrpKc { double lnA, n, mC, lnAb, nb, mCb, A; int mode, np, nusum, idx, pw, nusumh; int nuh[8]; signed char sp[8], "
         "anu[8]; };\n__device__ const GrpKc GRP_KC[" << std::max<size_t>(kc.size(), 1) << "] = {\n";
    auto lnA = [](const RateConstHost& rc) { return rc.A > 0.0 ? std::log(rc.A) : -1.0e300; };
    for (auto& k : kc) {
        const ReactionHost& r = mh.reactions[k.ir];
        o << "  {" << lit(lnA(r.frc)) << ", " << lit(r.frc.n) << ", " << lit(-r.frc.C) << ", " << lit(lnA(r.brc)) << ", "
          << lit(r.brc.n) << ", " << lit(-r.brc.C) << ", " << lit(r.frc.A) << ", " << k.mode << ", " << k.np << ", " << k.nusum
          << ", " << k.ir << ", " << k.pw << ", (int)" << high((double)k.nusum) << "u, {";
        for (int j = 0; j < k.np; ++j) o << (j ? ", " : "") << "(int)" << high((double)k.parts[j].nu) << "u";
        o << (k.np ? "}, {" : "0}, {");
        for (int j = 0; j < k.np; ++j) o << (j ? ", " : "") << k.parts[j].isp;
        o << (k.np ? "}, {" : "0}, {");
        for (int j = 0; j < k.np; ++j) o << (j ? ", " : "") << k.parts[j].nu;
        o << (k.np ? "}},\n" : "0}},\n");
    }
    if (kc.empty()) o << "  {}\n";
    o << "};\n";
    // tick rates, by the number of factors
    std::vector<int> order(nr);
    for (int i = 0; i < nr; ++i) order[i] = i;
    auto rx_key = [&](int ir) {
        const ReactionHost& r = mh.reactions[ir];
        return std::make_tuple(!r.collider, r.reac.size(), r.prod.size());
    };
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return rx_key(a) < rx_key(b); });
    o << "__device__ const __align__(16) uint4 GRP_RX[" << nr << "] = {\n";
    for (int ir : order) {
        const ReactionHost& r = mh.reactions[ir];
        unsigned sp[2] = {0, 0}, co = (unsigned)r.reac.size() | (unsigned)r.prod.size() << 3;
        int side = 0;
        for (auto* v : {&r.reac, &r.prod}) {
            for (size_t k = 0; k < v->size(); ++k) {
                sp[side] |= (unsigned)(*v)[k].first << (8 * k);
                co |= (unsigned)(*v)[k].second << (6 + 12 * side + 3 * k);
            }
            ++side;
        }
        o << "  {" << sp[0] << "u, " << sp[1] << "u, " << co << "u, "
          << ((unsigned)ir | (unsigned)(r.collider ? set_of[ir] + 1 : 0) << 16) << "u},\n";
    }
    o << "};\n__device__ const double GRP_EFF[" << std::max<size_t>(sets.size(), 1) * nsp << "] = {";
    for (auto& st : sets) {
        std::vector<double> e(nsp, 0.0);
        for (auto& x : st) e[x.first] = x.second;
        for (double v : e) o << lit(v) << ", ";
    }
    if (sets.empty()) o << "0.0";
    o << "};\n";
    if (nfall) {
        o << "__device__ const double GRP_FALL_EFF[" << nfall * nsp << "] = {";
        for (auto& r : mh.reactions) {
            if (!r.frc.pressure_dependent()) continue;
            std::vector<double> e(nsp, 0.0);
            for (auto& x : r.eff) e[x.first] = x.second;
            for (double v : e) o << lit(v) << ", ";
        }
        o << "};\n";
    }
    // q and L: q gets nu w_f (nu > 0) or -nu w_b, L gets nu w_b or -nu w_f (reaction_mechanism.d:82-96)
    std::vector<std::vector<std::pair<int, int>>> task(2 * nsp);
    for (int ir = 0; ir < nr; ++ir)
        for (auto& pp : participants(mh.reactions[ir])) {
            if (pp.nu == 0) continue;
            task[2 * pp.isp].push_back({pp.nu > 0 ? ir : nr + ir, std::abs(pp.nu)});
            task[2 * pp.isp + 1].push_back({pp.nu > 0 ? nr + ir : ir, std::abs(pp.nu)});
        }
    // RKF: index | coefficient << 16; alpha-QSS: index | log2 of the coefficient << 16, a coefficient that is no power
    // of two in several entries
    std::vector<std::vector<unsigned>> entries(2 * nsp);
    size_t n_ent = 0;
    for (int t = 0; t < 2 * nsp; ++t) {
        for (auto& e : task[t]) {
            if (mh.method == METHOD_RKF) entries[t].push_back((unsigned)e.first | (unsigned)e.second << 16);
            else
                for (int k = 0; k < 3; ++k)
                    if (e.second >> k & 1) entries[t].push_back((unsigned)e.first | (unsigned)k << 16);
        }
        n_ent += entries[t].size();
    }
    const size_t ent_size = (std::max<size_t>(n_ent, 1) + 1) & ~(size_t)1;
    o << "__device__ const __align__(16) unsigned GRP_ENT[" << ent_size << "] = {0u";
    {
        std::ostringstream es;
        for (auto& t : entries)
            for (unsigned e : t) es << (es.tellp() > 0 ? ", " : "") << e << "u";
        if (n_ent) { o.seekp(-2, std::ios_base::end); o << es.str(); }
    }
    o << "};\n__device__ const __align__(16) int GRP_TASK[" << ((2 * nsp + 1 + 1) & ~1) << "] = {0";
    size_t at = 0;
    for (auto& t : entries) o << ", " << (at += t.size());
    o << "};\n";
    std::vector<int> by_length(2 * nsp);
    for (int t = 0; t < 2 * nsp; ++t) by_length[t] = t;
    std::stable_sort(by_length.begin(), by_length.end(),
                     [&](int a, int b) { return entries[a].size() > entries[b].size(); });
    std::ostringstream starts, tasks;
    for (int lanes : {4, 8, 16, 32}) {
        std::vector<std::vector<int>> of(lanes);
        std::vector<size_t> load(lanes, 0);
        for (int t : by_length) {
            const int l = (int)(std::min_element(load.begin(), load.end()) - load.begin());
            of[l].push_back(t);
            load[l] += entries[t].size() + (mh.method == METHOD_RKF ? 1 : 2);
        }
        int n = 0;
        for (int l = 0; l < 33; ++l) {
            starts << (starts.tellp() > 0 ? ", " : "") << n;
            if (l < lanes) {
                for (int t : of[l]) tasks << (tasks.tellp() > 0 ? ", " : "") << t;
                n += (int)of[l].size();
            }
        }
    }
    o << "__device__ const __align__(16) int GRP_LANE_START[132] = {" << starts.str() << "};\n";
    o << "__device__ const __align__(16) int GRP_LANE_TASK[" << 8 * nsp << "] = {" << tasks.str() << "};\n";
    // the staged tables (GRP_TABLES of chem_group.cuh, checked there)
    shape.table_doubles = 2 * nr + nsp * 120 + GDTK_EXP2_TABLE_SIZE + std::max(nsets, 1) * nsp +
                          16 * (int)std::max<size_t>(kc.size(), 1) + (int)ent_size / 2 + (2 * nsp + 2) / 2 + 66 +
                          4 * nsp;
    o << "#define GDTK_GRP_CELL " << shape.cell_doubles << "\n#define GDTK_GRP_TABLES " << shape.table_doubles << "\n";
    return o.str();
}

std::string generate_fast_source(const GasModelHost& gm, const MechanismHost& mh, int block, int min_blocks,
                                 GroupShape* group_shape) {
    if (gm.n_species() > GDTK_MAX_SPECIES || (int)mh.reactions.size() > GDTK_MAX_REACTIONS)
        throw NoFastKernel("the mechanism-specialised kernel takes up to " + std::to_string(GDTK_MAX_SPECIES) +
                                 " species and " + std::to_string(GDTK_MAX_REACTIONS) +
                                 " reactions; larger mechanisms run one warp per cell");
    const int nsp = gm.n_species();
    const int nr = (int)mh.reactions.size();
    std::ostringstream o;
    o << "// generated: " << nsp << " species, " << nr << " reactions\n";
    o << "#define GDTK_NSP " << nsp << "\n#define GDTK_NR " << nr << "\n";
    o << "#define GDTK_METHOD " << mh.method << "\n#define GDTK_TIGHT " << (mh.tight ? 1 : 0) << "\n";
    o << "#define GDTK_MAX_ITERS " << mh.maxIters << "\n#define GDTK_MAX_SUBCYCLES " << mh.maxSubcycles << "\n";
    o << "#define GDTK_MAX_ATTEMPTS " << mh.maxAttempts << "\n";
    o << "#define GDTK_T_LOWER " << lit(mh.T_lower) << "\n#define GDTK_T_UPPER " << lit(mh.T_upper) << "\n";
    o << "#define GDTK_LN_T_LOWER " << lit(std::log(mh.T_lower)) << "\n#define GDTK_LN_T_UPPER "
      << lit(std::log(mh.T_upper)) << "\n";
    o << "#define GDTK_ERRTOL " << lit(mh.errTol) << "\n#define GDTK_EPS1 " << lit(mh.eps1) << "\n";
    o << "#define GDTK_EPS2 " << lit(mh.eps2) << "\n#define GDTK_DELTA " << lit(mh.delta) << "\n";
    o << "#define GDTK_BLOCK " << block << "\n#define GDTK_MIN_BLOCKS " << min_blocks << "\n";
    {
        double tlo = 0.0, thi = 0.0;
        const bool mix = mix_thermo_range(gm, tlo, thi);
        o << "#define GDTK_MIX_THERMO " << (mix ? 1 : 0) << "\n";
        if (mix) o << "#define GDTK_MIX_TLO " << lit(tlo) << "\n#define GDTK_MIX_THI " << lit(thi) << "\n";
        o << "#define GDTK_VEC " << fast_vec_doubles(gm, mh) << "\n";
        o << "#define GDTK_G_UNROLL _Pragma(\"unroll " << g_unroll() << "\")\n";
        const char* pc = std::getenv("GDTK_PHASE_CLOCKS");
        o << "#define GDTK_PHASE_CLOCKS " << ((pc && pc[0] == '1') ? 1 : 0) << "\n";
    }
    // one copy of exp and the division: fetching an inlined copy at each of some 30 places costs more than the calls
    // (262,147 H2-air cells 412 -> 393 ms, 9,001 methane cells 429 -> 384 ms), and half the compile time
    o << "#define GDTK_FN static __device__ __noinline__\n";
    o << kFastExpSource << "\n" << kCeaPolySource << "\n";
    auto arr = [&](const char* name, std::function<double(int)> f) {
        o << "__constant__ double " << name << "[" << nsp << "] = {";
        for (int i = 0; i < nsp; ++i) o << (i ? ", " : "") << lit(f(i));
        o << "};\n";
    };
    arr("GDTK_M", [&](int i) { return gm.M[i]; });
    arr("GDTK_RM", [&](int i) { return 1.0 / gm.M[i]; });
    arr("GDTK_R", [&](int i) { return R_universal / gm.M[i]; });
    o << "namespace gdtk_fast {\nusing gdtk::gdtk_exp;\nusing gdtk::gdtk_div;\nusing gdtk::gdtk_log;\nusing gdtk::gdtk_rcp;\n";

    // ---- third-body concentrations of the pressure-dependent rate constants (rate_constant.d:114-121),
    // from the concentrations at which the rate constants are evaluated
    int nfall = 0;
    o << "__device__ __forceinline__ void gen_falloff_M(const double (&c)[GDTK_NSP], double* Mv, int ms) {\n";
    o << "  (void)c; (void)Mv; (void)ms;\n";
    for (int ir = 0; ir < nr; ++ir) {
        const ReactionHost& r = mh.reactions[ir];
        if (!r.frc.pressure_dependent()) continue;
        o << "  { double m = 0.0;";
        for (auto& e : r.eff) o << " m = fma(" << lit(e.second) << ", c[" << e.first << "], m);";
        o << " Mv[" << nfall << " * ms] = m; }\n";
        ++nfall;
    }
    o << "}\n#define GDTK_NFALLOFF " << nfall << "\n";

    // ---- rate constants.  In table form (the default) the Arrhenius reactions are one loop over a
    // __constant__ table, which keeps the code the warps cycle through each step small (the kernel is
    // otherwise often stalled on instruction fetch); pressure-dependent reactions stay unrolled.
    const char* kc_env = std::getenv("GDTK_KC_UNROLLED");
    const bool kc_table = !(kc_env && kc_env[0] == '1');
    std::vector<int> table_rx;
    // 256 records of 208 bytes = 53 KB of the 64 KB constant bank, leaving room for the species constants;
    // reactions beyond them stay straight-line
    for (int ir = 0; ir < nr && (int)table_rx.size() < 256; ++ir) {
        const ReactionHost& r = mh.reactions[ir];
        int np = 0;
        for (auto& pp : participants(r)) np += pp.nu != 0;
        // the table holds ln A, n, C records; Arrhenius2 rate constants stay straight-line
        const bool arr2 = r.frc.model == RATE_ARRHENIUS2 || r.brc.model == RATE_ARRHENIUS2;
        if (kc_table && !r.frc.pressure_dependent() && !arr2 && np <= 8) table_rx.push_back(ir);
    }
    const std::vector<bool> kbp = kb_product_reactions(gm, mh);
    bool any_kbp = false;
    for (int ir : table_rx) any_kbp = any_kbp || kbp[ir];
    if (!table_rx.empty()) {
        // pw: k_f = A T^pw by multiplication (C = 0, integer |n| <= 4); 99: by exp of its logarithm
        o << "struct KcRec { double lnA, n, mC, lnAb, nb, mCb, A; int mode, np, nusum, idx, pw; int sp[8], anu[8]; "
             "double nu[8]; };\n";
        o << "__constant__ KcRec GDTK_KC_TAB[" << table_rx.size() << "] = {\n";
        for (int ir : table_rx) {
            const ReactionHost& r = mh.reactions[ir];
            auto parts = participants(r);
            int np = 0, nusum = 0;
            std::ostringstream sp, nu, anu;
            for (auto& pp : parts) {
                if (pp.nu == 0) continue;
                sp << (np ? ", " : "") << pp.isp;
                nu << (np ? ", " : "") << lit((double)pp.nu);
                anu << (np ? ", " : "") << pp.nu;   // signed: > 0 products, < 0 reactants
                nusum += pp.nu;
                ++np;
            }
            if (np == 0) { sp << "0"; nu << "0.0"; anu << "0"; }
            // mode 0: k_f Arrhenius, k_b from K_c; 1: both Arrhenius; 2: k_b Arrhenius, k_f from K_c;
            // 3: as 0, with k_b = k_f / K_c from the species' E_i
            int mode = r.frc.model == RATE_ARRHENIUS ? (r.brc.model == RATE_FROM_EQ ? 0 : 1) : 2;
            if (mode == 0 && kbp[ir]) mode = 3;
            auto lnA = [](const RateConstHost& rc) { return rc.A > 0.0 ? std::log(rc.A) : -1.0e300; };
            std::string pws;
            const int pw = power_arrhenius(r.frc, pws) ? (int)r.frc.n : 99;
            o << "  {" << lit(lnA(r.frc)) << ", " << lit(r.frc.n) << ", " << lit(-r.frc.C) << ", " << lit(lnA(r.brc))
              << ", " << lit(r.brc.n) << ", " << lit(-r.brc.C) << ", " << lit(r.frc.A) << ", " << mode << ", " << np
              << ", " << nusum << ", " << ir << ", " << pw << ", {" << sp.str() << "}, {" << anu.str() << "}, {"
              << nu.str() << "}},   // "
              << (r.equation.empty() ? std::string("reaction") : r.equation) << "\n";
        }
        o << "};\n";
    }
    o << "#define GDTK_LN_PATM_R " << lit(std::log(101325.0 / R_universal)) << "\n";
    o << "#define GDTK_R_PATM " << lit(R_universal / 101325.0) << "\n#define GDTK_PATM_R " << lit(101325.0 / R_universal) << "\n";
    if (nfall) {
        o << kFalloffSource << "__device__ const FallRec GDTK_FALL_TAB[" << nfall << "] = {\n";
        for (int ir = 0; ir < nr; ++ir)
            if (mh.reactions[ir].frc.pressure_dependent()) o << falloff_record(mh.reactions[ir], ir);
        o << "};\n";
    }
    o << "__device__ __forceinline__ void gen_kc(double T, double lnT, double rT, const double* g, int gs, double* K, "
         "int ks, const uint64_t* etab, const double* Mv, int ms) {\n";
    o << "  (void)T; (void)Mv; (void)ms;\n";
    if (any_kbp) {   // E_i = exp(G_i / R T) and its reciprocal, after G/RT and the falloff concentrations
        o << "  const double* E = g + (" << nsp << " + " << nfall << ") * gs;\n";
        o << "  const double* Ei = E + " << nsp << " * gs;\n";
        o << "#pragma unroll 1\n";
        o << "  for (int i = 0; i < " << nsp << "; ++i) {\n";
        o << "    const double e = gdtk_exp(g[i * gs], etab);\n";
        o << "    const_cast<double*>(E)[i * gs] = e;\n";
        o << "    const_cast<double*>(Ei)[i * gs] = gdtk_rcp(e);\n  }\n";
        o << "  const double cf = T * " << lit(R_universal / 101325.0) << ", rcf = rT * " << lit(101325.0 / R_universal)
          << ";   // R T / P_atm and its reciprocal\n";
    }
    if (!table_rx.empty()) {
        o << "#pragma unroll " << kc_unroll() << "\n";
        o << "  for (int t = 0; t < " << table_rx.size() << "; ++t) {   // reaction.d:26-52, 94-143\n";
        o << "    const KcRec& R = GDTK_KC_TAB[t];\n";
        if (any_kbp) {
            o << "    if (R.mode == 3) {   // k_b = k_f (R T / P_atm)^(sum nu) prod E_i^nu_i\n";
            o << "      double kf;\n";
            o << "      if (R.pw != 99) {   // A T^n, C = 0, integer n\n";
            o << "        const double b = R.pw > 0 ? T : rT;\n        kf = R.A;\n";
            o << "        for (int m = 0; m < abs(R.pw); ++m) kf *= b;\n";
            o << "      } else {\n        kf = gdtk_exp(fma(R.mC, rT, fma(R.n, lnT, R.lnA)), etab);\n      }\n";
            o << "      double P = 1.0;\n";
            o << "      const double c = R.nusum > 0 ? cf : rcf;\n";
            o << "      for (int m = 0; m < abs(R.nusum); ++m) P *= c;\n";
            o << "      for (int k = 0; k < R.np; ++k) {\n";
            o << "        const int nk = R.anu[k];\n";
            o << "        const double v = (nk > 0 ? E : Ei)[R.sp[k] * gs];\n";
            o << "        for (int m = 0; m < abs(nk); ++m) P *= v;\n      }\n";
            o << "      K[R.idx * ks] = kf;\n      K[(" << nr << " + R.idx) * ks] = kf * P;\n      continue;\n    }\n";
        }
        bool all_kbp = true;
        for (int ir : table_rx) all_kbp = all_kbp && kbp[ir];
        if (all_kbp) o << "#if 0   // every table reaction takes the product form\n";
        o << "    double dg = 0.0;\n";
        o << "    for (int k = 0; k < R.np; ++k) dg = fma(R.nu[k], g[R.sp[k] * gs], dg);\n";
        o << "    const double lnKc = fma((double)R.nusum, " << lit(std::log(101325.0 / R_universal)) << " - lnT, -dg);\n";
        o << "    double kf, kb;\n";
        o << "    if (R.mode != 2) {\n";
        o << "      const double lkf = fma(R.mC, rT, fma(R.n, lnT, R.lnA));\n";
        o << "      kf = gdtk_exp(lkf, etab);\n";
        o << "      kb = R.mode == 0 ? gdtk_exp(lkf - lnKc, etab) : gdtk_exp(fma(R.mCb, rT, fma(R.nb, lnT, R.lnAb)), etab);\n";
        o << "    } else {\n";
        o << "      const double lkb = fma(R.mCb, rT, fma(R.nb, lnT, R.lnAb));\n";
        o << "      kb = gdtk_exp(lkb, etab);\n";
        o << "      kf = gdtk_exp(lkb + lnKc, etab);\n";
        o << "    }\n";
        o << "    K[R.idx * ks] = kf;\n    K[(" << nr << " + R.idx) * ks] = kb;\n";
        if (all_kbp) o << "#endif\n";
        o << "  }\n";
    }
    if (nfall) {
        o << "#pragma unroll 1\n  for (int f = 0; f < " << nfall << "; ++f) {\n    double kf, kb;\n";
        o << "    falloff_rates(GDTK_FALL_TAB[f], T, lnT, rT, Mv[f * ms], g, gs, etab, kf, kb);\n";
        o << "    K[GDTK_FALL_TAB[f].idx * ks] = kf;\n    K[(" << nr << " + GDTK_FALL_TAB[f].idx) * ks] = kb;\n  }\n";
    }
    for (int ir = 0; ir < nr; ++ir) {
        const ReactionHost& r = mh.reactions[ir];
        if (r.frc.pressure_dependent() || std::find(table_rx.begin(), table_rx.end(), ir) != table_rx.end()) continue;
        auto parts = participants(r);
        if (ir > 0 && ir % 4 == 0) o << "  asm volatile(\"\" ::: \"memory\");\n";
        std::string dgs = "0.0";   // sum nu * G/RT
        int nusum = 0;
        for (auto& p : parts) {
            if (p.nu == 0) continue;
            nusum += p.nu;
            dgs = "fma(" + lit((double)p.nu) + ", g[" + std::to_string(p.isp) + " * gs], " + dgs + ")";
        }
        // ln K_c = -sum(nu G/RT) + sum(nu) ln(P_atm / R T)   (reaction.d:26-52)
        std::string lnKc = "(-(" + dgs + ")" +
                           (nusum ? " + " + lit((double)nusum) + " * (" + lit(std::log(101325.0 / R_universal)) + " - lnT)" : std::string("")) + ")";
        o << "  { // " << (r.equation.empty() ? std::string("reaction") : r.equation) << "\n";
        if (r.frc.simple()) {
            std::string pw;
            if (power_arrhenius(r.frc, pw)) {
                o << "    const double kf = " << pw << ";\n";
                if (r.brc.model == RATE_FROM_EQ) o << "    const double kb = kf * gdtk_exp(-" << lnKc << ", etab);\n";
            } else {
                std::string l = log_arrhenius(r.frc);
                if (l.empty()) o << "    const double lkf = -1.0e300; const double kf = 0.0;\n";
                else o << "    const double lkf = " << l << ";\n    const double kf = gdtk_exp(lkf, etab);\n";
                if (r.brc.model == RATE_FROM_EQ) o << "    const double kb = gdtk_exp(lkf - " << lnKc << ", etab);\n";
            }
            if (r.brc.simple()) {
                std::string pb;
                if (power_arrhenius(r.brc, pb)) o << "    const double kb = " << pb << ";\n";
                else {
                    std::string l = log_arrhenius(r.brc);
                    o << "    const double kb = " << (l.empty() ? std::string("0.0") : "gdtk_exp(" + l + ", etab)")
                      << ";\n";
                }
            }
        } else {   // forward from K_c and a given backward rate constant
            std::string l = log_arrhenius(r.brc);
            if (l.empty()) o << "    const double kb = 0.0; const double kf = 0.0;\n";
            else o << "    const double lkb = " << l << ";\n    const double kb = gdtk_exp(lkb, etab);\n"
                   << "    const double kf = gdtk_exp(lkb + " << lnKc << ", etab);\n";
        }
        o << "    K[" << ir << " * ks] = kf;\n    K[" << (nr + ir) << " * ks] = kb;\n  }\n";
    }
    o << "}\n";

    // ---- production / loss rates
    o << "__device__ __forceinline__ void gen_rhs(const double* c, double* q, double* L, const double* K, int ks) {\n";
    // distinct third-body lists
    std::vector<std::vector<std::pair<int, double>>> sets;
    std::vector<int> set_of(nr, -1);
    for (int ir = 0; ir < nr; ++ir) {
        const ReactionHost& r = mh.reactions[ir];
        if (!r.collider) continue;
        int f = -1;
        for (size_t s = 0; s < sets.size(); ++s) if (sets[s] == r.eff) { f = (int)s; break; }
        if (f < 0) { sets.push_back(r.eff); f = (int)sets.size() - 1; }
        set_of[ir] = f;
    }
    for (size_t s = 0; s < sets.size(); ++s) {
        std::vector<double> leaf(nsp, 0.0);
        for (auto& e : sets[s]) leaf[e.first] = e.second;
        int p2 = 1;
        while (p2 < nsp) p2 *= 2;
        const std::string sum = third_body_sum(leaf, 0, p2);
        o << "  const double M" << s << " = " << (sum.empty() ? "0.0" : sum) << ";\n";
    }
    std::vector<bool> qset(nsp, false), lset(nsp, false);
    auto acc = [&](std::vector<bool>& set, const char* arr, int isp, int coeff, const char* w) {
        std::string dst = std::string(arr) + "[" + std::to_string(isp) + "]";
        std::string val = coeff == 1 ? std::string(w) : lit((double)coeff) + " * " + w;
        if (!set[isp]) { o << "    " << dst << " = " << val << ";\n"; set[isp] = true; }
        else if (coeff == 1) o << "    " << dst << " += " << w << ";\n";
        else o << "    " << dst << " = fma(" << lit((double)coeff) << ", " << w << ", " << dst << ");\n";
    };
    for (int ir = 0; ir < nr; ++ir) {
        const ReactionHost& r = mh.reactions[ir];
        // A compiler barrier every few reactions stops the scheduler from hoisting every k_f/k_b
        // load to the top, which would hold 2 NR doubles live and spill registers.
        if (ir > 0 && rhs_fence() > 0 && ir % rhs_fence() == 0) o << "  asm volatile(\"\" ::: \"memory\");\n";
        o << "  {\n    double wf = K[" << ir << " * ks], wb = K[" << (nr + ir) << " * ks];\n";
        if (r.collider) o << "    wf *= M" << set_of[ir] << "; wb *= M" << set_of[ir] << ";\n";
        // products that the compiler may not contract into the sums: the same rates in every kernel
        for (auto& x : r.reac) o << "    wf = __dmul_rn(wf, " << ipow_expr("c[" + std::to_string(x.first) + "]", x.second) << ");\n";
        for (auto& x : r.prod) o << "    wb = __dmul_rn(wb, " << ipow_expr("c[" + std::to_string(x.first) + "]", x.second) << ");\n";
        for (auto& p : participants(r)) {
            if (p.nu > 0) { acc(qset, "q", p.isp, p.nu, "wf"); acc(lset, "L", p.isp, p.nu, "wb"); }
            else if (p.nu < 0) { acc(qset, "q", p.isp, -p.nu, "wb"); acc(lset, "L", p.isp, -p.nu, "wf"); }
        }
        o << "  }\n";
    }
    for (int i = 0; i < nsp; ++i) {
        if (!qset[i]) o << "  q[" << i << "] = 0.0;\n";
        if (!lset[i]) o << "  L[" << i << "] = 0.0;\n";
    }
    o << "}\n";
    const bool group = group_kernel_takes(mh, table_rx.size(), (size_t)nfall);
    o << "#define GDTK_GROUP " << (group ? 1 : 0) << "\n";
    GroupShape shape;
    if (group) o << group_tables(gm, mh, table_rx, kbp, sets, set_of, shape);
    if (group_shape) *group_shape = shape;
    o << "}  // namespace gdtk_fast\n";
    o << kFastCuhSource;
    if (group) o << kGroupCuhSource;
    return o.str();
}

namespace {

std::string cache_dir() {
    const char* env = std::getenv("GDTK_JIT_CACHE");
    if (env && *env) return env;
    const char* home = std::getenv("HOME");
    return std::string(home && *home ? home : "/tmp") + "/.cache/gdtk_gb300";
}

std::string arch_option(int major, int minor) {
    return "--gpu-architecture=sm_" + std::to_string(major) + std::to_string(minor) + (major >= 9 ? "a" : "");
}
const char* const kJitOptions[] = {"--std=c++17", "--fmad=true", "-default-device", "-lineinfo",
                                   "--ptxas-options=-v"};

// Key of the in-process and on-disk cubin caches: the source, the target, NVRTC's version and
// every compile option, so a toolkit upgrade or an option change never loads a stale cubin.
std::string cubin_cache_key(const std::string& src, int major, int minor) {
    int vmaj = 0, vmin = 0;
    nvrtcVersion(&vmaj, &vmin);
    std::string opts = arch_option(major, minor);
    for (const char* o : kJitOptions) opts += std::string(" ") + o;
    const size_t h = std::hash<std::string>{}(src) ^ (std::hash<std::string>{}(opts) * 0x9e3779b97f4a7c15ull);
    return std::to_string(h) + "_sm" + std::to_string(major) + std::to_string(minor) + "_nvrtc" +
           std::to_string(vmaj) + "." + std::to_string(vmin);
}

std::string compile_cubin(const std::string& src, int major, int minor, std::string& log) {
    const std::string arch = arch_option(major, minor);
    std::vector<const char*> opts{arch.c_str()};
    for (const char* o : kJitOptions) opts.push_back(o);
    nvrtcProgram prog;
    if (nvrtcCreateProgram(&prog, src.c_str(), "gdtk_chem_fast.cu", 0, nullptr, nullptr) != NVRTC_SUCCESS)
        throw std::runtime_error("nvrtcCreateProgram failed");
    nvrtcResult rc = nvrtcCompileProgram(prog, (int)opts.size(), opts.data());
    size_t n = 0;
    nvrtcGetProgramLogSize(prog, &n);
    log.assign(n, '\0');
    if (n) nvrtcGetProgramLog(prog, &log[0]);
    while (!log.empty() && log.back() == '\0') log.pop_back();
    if (rc != NVRTC_SUCCESS) {
        nvrtcDestroyProgram(&prog);
        const std::string why = std::string("NVRTC compilation of the mechanism kernel failed: ") + nvrtcGetErrorString(rc) + "\n" + log;
        if (rc == NVRTC_ERROR_COMPILATION) throw NoFastKernel(why);
        throw std::runtime_error(why);
    }
    size_t cn = 0;
    nvrtcGetCUBINSize(prog, &cn);
    std::string cubin(cn, '\0');
    nvrtcGetCUBIN(prog, &cubin[0]);
    nvrtcDestroyProgram(&prog);
    return cubin;
}

std::mutex g_jit_mu;
std::map<std::string, std::string> g_cubins;   // source hash key -> cubin (this process)

}  // namespace

std::string compile_fast_check(const GasModelHost& gm, const MechanismHost& mh, int major, int minor) {
    std::string log;
    std::string src = generate_fast_source(gm, mh, 256, 1);
    std::string cubin = compile_cubin(src, major, minor, log);
    return log + "\ncubin bytes: " + std::to_string(cubin.size()) + "\n";
}

static size_t group_smem(const GroupShape& g, int block, int lanes) {
    return (size_t)(g.table_doubles + g.cell_doubles * (block / lanes)) * 8;
}

FastKernel* build_fast_kernel(const GasModelHost& gm, const MechanismHost& mh, int req_block, int req_min_blocks) {
    int dev = 0, major = 0, minor = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
    cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int nsp = gm.n_species(), nr = (int)mh.reactions.size();
    if (nsp > GDTK_MAX_SPECIES || nr > GDTK_MAX_REACTIONS) generate_fast_source(gm, mh, 32, 1);   // throws the reason
    const int per_thread = 2 * nr + fast_vec_doubles(gm, mh);
    const int table = nsp * 120 + GDTK_EXP2_TABLE_SIZE;
    // Block size: as many resident threads as shared memory allows, up to 256 per SM.  Each resident
    // block also holds the kernel's static shared arrays (at most kStaticSmem bytes, the phase-clock
    // instrumentation) and the 1 KB the hardware reserves per block; one block may use up to 227 KB.
    constexpr double kStaticSmem = 512.0, kReserved = 1024.0, kSmPerSm = 228.0 * 1024, kSmPerBlock = 227.0 * 1024;
    auto fits = [&](int blk, int nblk) {
        const double dyn = (table + (double)per_thread * blk) * 8.0;
        return dyn + kStaticSmem <= kSmPerBlock && nblk * (dyn + kStaticSmem + kReserved) <= kSmPerSm;
    };
    int block = 256, min_blocks = 1;
    while (block > 32 && !fits(block, 1)) block -= 32;
    if (!fits(block, 1)) throw NoFastKernel("mechanism too large for shared memory");
    if (block <= 128 && fits(block, 2)) min_blocks = 2;
    if (req_block > 0) {   // an explicit launch shape (autotuning)
        if (req_block % 32 || req_block > 1024) throw std::runtime_error("block size must be a multiple of 32, <= 1024");
        int mb = req_min_blocks > 0 ? req_min_blocks : 1;
        if (!fits(req_block, mb)) throw std::runtime_error("requested block shape does not fit in shared memory");
        block = req_block;
        min_blocks = mb;
    }

    auto k = std::make_unique<FastKernel>();
    k->block = block;
    k->min_blocks = min_blocks;
    k->method = mh.method;
    k->per_thread_doubles = per_thread;
    k->table_doubles = table;
    k->source = generate_fast_source(gm, mh, block, min_blocks, &k->group);
    std::string key = cubin_cache_key(k->source, major, minor);
    std::string cubin;
    {
        std::lock_guard<std::mutex> lk(g_jit_mu);
        auto it = g_cubins.find(key);
        if (it != g_cubins.end()) cubin = it->second;
    }
    std::string dir = cache_dir(), path = dir + "/" + key + ".cubin";
    if (cubin.empty()) {
        std::ifstream f(path, std::ios::binary);
        if (f) {
            std::ostringstream ss;
            ss << f.rdbuf();
            cubin = ss.str();
            k->log = "loaded from " + path;
        }
    }
    if (cubin.empty()) {
        cubin = compile_cubin(k->source, major, minor, k->log);
        std::string tmp = path + ".tmp" + std::to_string((long)getpid());
        ::mkdir((dir.substr(0, dir.rfind('/'))).c_str(), 0755);
        ::mkdir(dir.c_str(), 0755);
        std::ofstream f(tmp, std::ios::binary);
        if (f) {
            f.write(cubin.data(), (std::streamsize)cubin.size());
            f.close();
            std::rename(tmp.c_str(), path.c_str());
        }
    }
    Driver& d = driver();
    CUmodule mod;
    cu_check(d.moduleLoadData(&mod, cubin.data()), "cuModuleLoadData");
    k->module = mod;
    {   // one that loads
        std::lock_guard<std::mutex> lk(g_jit_mu);
        g_cubins[key] = cubin;
    }
    CUfunction fn;
    cu_check(d.moduleGetFunction(&fn, mod, "gdtk_chem_fast"), "cuModuleGetFunction");
    k->function = fn;
    CUfunction cfn;
    cu_check(d.moduleGetFunction(&cfn, mod, "gdtk_chem_cost"), "cuModuleGetFunction");
    k->cost_function = cfn;
    CUfunction sfn;
    cu_check(d.moduleGetFunction(&sfn, mod, "gdtk_chem_source"), "cuModuleGetFunction");
    k->source_function = sfn;
    const size_t smem_max = (size_t)(table + per_thread * block) * 8;
    cu_check(d.funcSetAttribute(sfn, CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES, (int)smem_max),
             "cuFuncSetAttribute");
    cu_check(d.funcSetAttribute(fn, CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES, (int)smem_max),
             "cuFuncSetAttribute");
    cu_check(d.funcSetAttribute(cfn, CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES, (int)smem_max),
             "cuFuncSetAttribute");
    cu_check(d.occupancy(&k->blocks_per_sm, fn, block, smem_max), "cuOccupancyMaxActiveBlocksPerMultiprocessor");
    if (k->blocks_per_sm < 1) throw NoFastKernel("fast kernel cannot be resident (registers/shared memory)");
    if (k->group.cell_doubles) {
        CUfunction gfn;
        cu_check(d.moduleGetFunction(&gfn, mod, "gdtk_chem_group"), "cuModuleGetFunction");
        cu_check(d.funcSetAttribute(gfn, CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES, (int)kSmPerBlock),
                 "cuFuncSetAttribute");
        // one block per SM: as many warps as its cells' slices fit beside the tables
        for (int lv = 0; lv < 4; ++lv) {
            int w = kGroupBlock / 32;
            while (w > 0 && group_smem(k->group, 32 * w, 4 << lv) > (size_t)kSmPerBlock) --w;
            k->group_warps[lv] = w;
        }
        k->group_function = gfn;
    }
    std::vector<double> th = fast_thermo_table(gm);
    static const uint64_t etab[GDTK_EXP2_TABLE_SIZE] = GDTK_EXP2_TABLE_INIT;
    // on a stream of its own: the default stream may not be used while another stream is captured
    cudaStream_t copies = nullptr;
    cudaError_t e = cudaStreamCreateWithFlags(&copies, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(&k->d_thermo, th.size() * 8);
    if (e == cudaSuccess) e = cudaMalloc(&k->d_exp, sizeof etab);
    if (e == cudaSuccess) e = cudaMemcpyAsync(k->d_thermo, th.data(), th.size() * 8, cudaMemcpyHostToDevice, copies);
    if (e == cudaSuccess) e = cudaMemcpyAsync(k->d_exp, etab, sizeof etab, cudaMemcpyHostToDevice, copies);
    if (e == cudaSuccess) e = cudaStreamSynchronize(copies);
    if (copies) cudaStreamDestroy(copies);
    if (e != cudaSuccess) throw std::runtime_error(std::string("tables of the mechanism kernel: ") + cudaGetErrorString(e));
    (void)sms;
    return k.release();
}

cudaError_t launch_fast(FastKernel& k, FastArgs& a, int sm_count, cudaStream_t stream, int* grid_out, int* block_out,
                        int* smem_out) {
    a.thermo = k.d_thermo;
    a.exp_table = k.d_exp;
    int block = k.block;
    while (block > 32 && ((long long)a.total + block - 1) / block < sm_count) block -= 32;
    long long want = ((long long)a.total + block - 1) / block;
    long long grid = (long long)sm_count * k.blocks_per_sm * (k.block / block);
    if (want < grid) grid = want;
    if (grid < 1) grid = 1;
    size_t smem = (size_t)(k.table_doubles + k.per_thread_doubles * block) * 8;
    void* params[] = {&a};
    CUresult r = driver().launchKernel((CUfunction)k.function, (unsigned)grid, 1, 1, (unsigned)block, 1, 1,
                                       (unsigned)smem, (CUstream)stream, params, nullptr);
    if (grid_out) *grid_out = (int)grid;
    if (block_out) *block_out = block;
    if (smem_out) *smem_out = (int)smem;
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorLaunchFailure;
}

// More lanes shorten a cell's step but spend more FP64 instructions on it (a cell's own scalars and sums are computed
// by every lane), so the most lanes are taken while the cells, in turns of the resident ones, do not
// exceed `turns`: measured where two choices cross.  H2-air (13 species; ms with 4 / 8 / 16 / 32 lanes): 1,000 cells
// 36 / 31 / 29 / 29, 12,000 63 / 52 / 48 / 54, 48,000 108 / 96 / 109 / 179, 262,147 364 / 437 / 575 / 975.  The
// Runge-Kutta mechanisms are smaller (5 species) and their cells' step counts alike, so that no long tail
// pays for lanes: 1,000 air cells 2.6 / 1.9 / 1.7 / 1.8, 4,000 2.9 / 2.3 / 2.7 / 3.6, 12,000 3.5 / 4.3 / 5.8 / 9.6.
// Against one thread per cell 4 lanes lie ahead for one turn, 19,456 cells: over 2e-7 s 2.9 and 4.1 at 12,000, 3.8 and 4.1 at
// 16,384, 3.9 and 4.0 at 19,000 (Gupta's air 11.6 and 12.5), 8.3 and 4.3 at 32,768.
int group_lanes(const FastKernel& k, long long total, int sm_count) {
    if (!k.group_function) return 0;
    const bool rkf = k.method == METHOD_RKF;
    const double turns[4] = {rkf ? 1.0 : 1e30, rkf ? 0.65 : 7.0, rkf ? 0.44 : 6.5, rkf ? 0.3 : 1.6};
    for (int lv = 3; lv >= 0; --lv) {
        const double resident = (double)sm_count * k.group_warps[lv] * (8 >> lv);
        if ((double)total <= turns[lv] * resident) return 4 << lv;
    }
    return 0;
}

cudaError_t launch_group(FastKernel& k, FastArgs& a, int lanes, int sm_count, cudaStream_t stream, int* grid_out,
                         int* block_out, int* smem_out) {
    a.thermo = k.d_thermo;
    a.exp_table = k.d_exp;
    int lv = 0;
    while ((4 << lv) < lanes) ++lv;
    // one block per SM, so that the tables are staged once per SM; the warps spread over all SMs
    const long long warps = ((long long)a.total * lanes + 31) / 32;
    const long long per_sm = std::min<long long>(std::max<long long>((warps + sm_count - 1) / sm_count, 1), k.group_warps[lv]);
    const int block = 32 * (int)per_sm;
    const long long grid = std::min<long long>((warps + per_sm - 1) / per_sm, sm_count);
    const size_t smem = group_smem(k.group, block, lanes);
    void* params[] = {&a, &lanes};
    CUresult r = driver().launchKernel((CUfunction)k.group_function, (unsigned)grid, 1, 1, (unsigned)block, 1, 1,
                                       (unsigned)smem, (CUstream)stream, params, nullptr);
    if (grid_out) *grid_out = (int)grid;
    if (block_out) *block_out = block;
    if (smem_out) *smem_out = (int)smem;
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorLaunchFailure;
}

cudaError_t launch_source(FastKernel& k, int n, const double* rho, const double* T, const double* massf, double* source,
                          int* status, int sm_count, cudaStream_t stream) {
    int block = k.block;
    while (block > 32 && ((long long)n + block - 1) / block < sm_count) block -= 32;
    const long long want = ((long long)n + block - 1) / block;
    const long long grid = std::min<long long>(want, (long long)sm_count * k.blocks_per_sm * (k.block / block));
    const size_t smem = (size_t)(k.table_doubles + k.per_thread_doubles * block) * 8;
    const double* thermo = k.d_thermo;
    const uint64_t* etab = k.d_exp;
    void* params[] = {&thermo, &etab, &n, &rho, &T, &massf, &source, &status};
    CUresult r = driver().launchKernel((CUfunction)k.source_function, (unsigned)grid, 1, 1, (unsigned)block, 1, 1,
                                       (unsigned)smem, (CUstream)stream, params, nullptr);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorLaunchFailure;
}

cudaError_t launch_order(FastKernel& k, FastArgs& a, int sm_count, float* key, int* order, int* hist,
                         cudaStream_t stream) {
    a.thermo = k.d_thermo;
    a.exp_table = k.d_exp;
    const int block = k.block;
    long long grid = ((long long)a.total + block - 1) / block;
    if (grid > (long long)sm_count * k.blocks_per_sm) grid = (long long)sm_count * k.blocks_per_sm;
    if (grid < 1) grid = 1;
    size_t smem = (size_t)(k.table_doubles + k.per_thread_doubles * block) * 8;
    void* params[] = {&a, &key};
    CUresult r = driver().launchKernel((CUfunction)k.cost_function, (unsigned)grid, 1, 1, (unsigned)block, 1, 1,
                                       (unsigned)smem, (CUstream)stream, params, nullptr);
    if (r != CUDA_SUCCESS) return cudaErrorLaunchFailure;
    return launch_bucket_order(key, a.total, order, hist, sm_count, stream);
}

}  // namespace gdtk

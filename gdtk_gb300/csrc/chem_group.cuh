// chem_group.cuh -- the chemistry update with a group of L lanes per cell (L = 4, 8, 16, 32).
//
// Compiled by NVRTC after the generated prologue and chem_fast.cuh, whose arithmetic it shares: a cell's
// result does not depend on L, bit for bit (sums over species take the same zero-padded pairwise tree, gathers
// the same ascending order of reactions), and for the Runge-Kutta method it is the one-thread-per-cell kernel's, so
// that the choice among them, made from the batch's size, never shows in a result.  The alpha-QSS method, whose
// q and L sums are rounded once here (grp_gather), takes a group for every size of batch.
//
// Why: an FP64 warp instruction costs 64 cycles (76 with all sub-partitions busy) however few of its lanes
// are active, so with one cell per lane a step of the 13-species, 33-reaction H2-air mechanism takes
// about 100 us, and a batch waits that long for each of the 2,000 steps of its longest cell.  Here a cell's
// species and reactions are spread over L lanes: the species' G/RT, exponentials and alpha-QSS updates, the
// reactions' rate constants and tick rates, and the q and L sums (dealt whole to the lanes, longest first).
// What is per cell (time step control, the Newton iteration) every lane of the group computes alike.
// A cell's vectors live in its group's slice of shared memory; the tables are staged there once per block.
//
// Warps keep all their groups in step (every __syncwarp and shuffle is over the whole warp, in loops that
// are uniform over it), because groups that drift apart would each issue their own FP64 instructions.
// When the queue of cells is empty and at most half of a warp's groups still hold one, the warp
// regroups: the cells left take twice the lanes each, up to all 32, which shortens the tail.

#if GDTK_GROUP
namespace gdtk_fast {

constexpr int pow2_at_least(int n) { int p = 1; while (p < n) p *= 2; return p; }
constexpr int GRP_P2 = pow2_at_least(GDTK_NSP);
constexpr int grp_max(int a, int b) { return a > b ? a : b; }

// a cell's slice of shared memory, in doubles
constexpr int GO_Y0 = 0, GO_C = GDTK_NSP, GO_Q = 2 * GDTK_NSP, GO_L = 3 * GDTK_NSP, GO_K = 4 * GDTK_NSP,
              GO_W = GO_K + 2 * GDTK_NR;   // tick rates; G/RT, E, 1/E, falloff [M]; Y_i R_i and mixture coefficients
constexpr int GO_M = GO_W + grp_max(2 * GDTK_NR, grp_max(3 * GDTK_NSP + GDTK_NFALLOFF, GDTK_NSP + 24));
constexpr int GO_V = GO_M + GDTK_NSETS;    // RKF: k1..k6; alpha-QSS: q0, p0 / 2, yp0
constexpr int GRP_CELL = (GO_V + (GDTK_METHOD == 0 ? 6 : 3) * GDTK_NSP) | 1;   // odd: slices start on different banks
static_assert(GRP_CELL == GDTK_GRP_CELL, "the host's size of a cell's slice");

constexpr int GRP_TABLES = (int)((sizeof GRP_RX + sizeof GRP_EFF + sizeof GRP_KC + sizeof GRP_ENT + sizeof GRP_TASK +
                                  sizeof GRP_LANE_START + sizeof GRP_LANE_TASK) / 8) + GDTK_NSP * GDTK_TH_STRIDE +
                           GDTK_EXP2_TABLE_SIZE;
static_assert(GRP_TABLES == GDTK_GRP_TABLES, "the host's size of the tables");

// The tables of a block, staged from GRP_TABLES (codegen.cpp) in this order.
struct GrpTab {
    const double* TH;
    const uint64_t* ETAB;
    const double* eff;        // [NSETS][NSP] third-body efficiencies, 0 where absent
    const GrpKc* kc;
    const uint4* rx;
    const unsigned* ent;      // the terms of the q and L sums, task by task: tick-rate index, coefficient (codegen.cpp)
    const int* task;          // first entry of each task (2 NSP + 1); task 2 i is q_i, 2 i + 1 L_i
    const int* lane_start;    // per L (4, 8, 16, 32): first slot of each lane (L + 1)
    const int* lane_task;     // per L: the tasks in lane order
};

struct GrpCell {
    double* S;                // the cell's slice
    unsigned g;
    int b, ci;
    bool have, retried, need_kc;
    int phase, cycle, attempt, err;
    double rho, rrho, u, T, lnT, p, dtS, dtS0, dtSave, h, t, tI;
    int n_steps, n_rhs, n_kc, n_newton, n_rej, n_est;
};

constexpr unsigned GRP_FULL = 0xffffffffu;

// e c with the roundings of the product, which most efficiencies, 1, do not need
__device__ __forceinline__ double third_body(double e, double c) { return dbits(e) == dbits(1.0) ? c : __dmul_rn(e, c); }
// x / 2 for x = 0 or normal x > 0
__device__ __forceinline__ double half_nn(double x) {
    return (unsigned long long)((dbits(x) >> 52) - 2) < 0x7fcULL ? __longlong_as_double(dbits(x) - (1LL << 52)) : 0.5 * x;
}

#if GDTK_METHOD == 0
__constant__ int GRP_COEF_HI[8] = {0, 0x3ff00000, 0x40000000, 0x40080000, 0x40100000, 0x40140000, 0x40180000, 0x401c0000};
#endif

// sum over the species of leaf(i), the zero-padded pairwise tree of sum_pairwise; every lane gets it.
template <int L, typename F>
__device__ __forceinline__ double grp_sum(int gl, F leaf) {
    constexpr int W = L < GRP_P2 ? L : GRP_P2, KC = GRP_P2 / W;
    const int base = (gl & (W - 1)) * KC;
    double v[KC];
#pragma unroll
    for (int k = 0; k < KC; ++k) v[k] = base + k < GDTK_NSP ? leaf(base + k) : 0.0;
#pragma unroll
    for (int w = 1; w < KC; w <<= 1)
#pragma unroll
        for (int k = 0; k < KC; k += 2 * w) v[k] += v[k + w];
#pragma unroll
    for (int x = 1; x < W; x <<= 1) v[0] += __shfl_xor_sync(GRP_FULL, v[0], x);
    return v[0];
}

// the largest ratio num / den of leaf(i), by the tree and the comparison of sigma_of
template <int L, typename F>
__device__ __forceinline__ Ratio grp_max_ratio(int gl, F leaf) {
    constexpr int W = L < GRP_P2 ? L : GRP_P2, KC = GRP_P2 / W;
    const int base = (gl & (W - 1)) * KC;
    Ratio v[KC];
#pragma unroll
    for (int k = 0; k < KC; ++k) v[k] = base + k < GDTK_NSP ? leaf(base + k) : Ratio{0.0, 1.0};
#pragma unroll
    for (int w = 1; w < KC; w <<= 1)
#pragma unroll
        for (int k = 0; k < KC; k += 2 * w) v[k] = larger_ratio(v[k], v[k + w]);
#pragma unroll
    for (int x = 1; x < W; x <<= 1) {
        Ratio o;
        o.num = __shfl_xor_sync(GRP_FULL, v[0].num, x);
        o.den = __shfl_xor_sync(GRP_FULL, v[0].den, x);
        v[0] = (gl & x) ? larger_ratio(o, v[0]) : larger_ratio(v[0], o);
    }
    return v[0];
}

// Rate constants at (T, ln T) into S[GO_K..] for the groups with `act` (rate_constants and gen_kc).
template <int L>
__device__ __forceinline__ void grp_rate_constants(const GrpTab& tab, GrpCell& s, int gl, bool act) {
    double* G = s.S + GO_W;
    double T = s.T, lnT = s.lnT;
    if (lt_pos(T, GDTK_T_LOWER)) { T = GDTK_T_LOWER; lnT = GDTK_LN_T_LOWER; }
    if (gt_pos(T, GDTK_T_UPPER)) { T = GDTK_T_UPPER; lnT = GDTK_LN_T_UPPER; }
    double rT = 0.0;
    int e = 0;
    if (act) {
        rT = gdtk_rcp(T);
        const double rT2 = rT * rT, t1 = lnT + 1.0, t2 = 1.0 - lnT;
        double* E = G + GDTK_NSP + GDTK_NFALLOFF;
#if GDTK_MIX_THERMO
        int sa = 0, sb = 0;
        double wb = 0.0;
        const bool mix = in_mix_range(T) && seg_of(tab.TH, T, sa, sb, wb);
#endif
#pragma unroll 1
        for (int i = gl; i < GDTK_NSP; i += L) {
            double g;
#if GDTK_MIX_THERMO
            if (mix) {
                const double* c = tab.TH + i * GDTK_TH_STRIDE + GDTK_TH_SEG0 + 15;
                g = poly_G(c + 24 * sa, T, rT, rT2, t1, t2);
                if (nonzero(wb)) g = fma(wb, poly_G(c + 24 * sb, T, rT, rT2, t1, t2) - g, g);
            } else
#endif
                g = sp_G(tab.TH, i, T, lnT, rT, rT2, t1, t2, e);
            G[i] = g;
#if GDTK_ANY_KBP
            const double x = gdtk_exp(g, tab.ETAB);
            E[i] = x;
            E[GDTK_NSP + i] = gdtk_rcp(x);
#endif
        }
        (void)E;
#if GDTK_NFALLOFF
        const double* c = s.S + GO_Y0;
#pragma unroll 1
        for (int f = gl; f < GDTK_NFALLOFF; f += L) {
            double M = 0.0;
#pragma unroll 7
            for (int i = 0; i < GDTK_NSP; ++i) {
                const double x = GRP_FALL_EFF[f * GDTK_NSP + i], y = fma(x, c[i], M);
                M = nonzero(x) ? y : M;
            }
            G[GDTK_NSP + f] = M;
        }
#endif
    }
    // an error of any lane is the group's
#pragma unroll
    for (int x = 1; x < L; x <<= 1) e |= __shfl_xor_sync(GRP_FULL, e, x);
    if (act && e) s.err = e;
    __syncwarp(GRP_FULL);
    if (act) {
        double* K = s.S + GO_K;
#if GDTK_ANY_KBP
        const double* E = G + GDTK_NSP + GDTK_NFALLOFF;
        const double cf = T * GDTK_R_PATM, rcf = rT * GDTK_PATM_R;
#endif
#pragma unroll 1
        for (int r = gl; r < GDTK_NKC; r += L) {
            const GrpKc& R = tab.kc[r];
            double kf, kb;
#if GDTK_ANY_KBP
            if (R.mode == 3) {
                if (R.pw != 99) {
                    const double b = R.pw > 0 ? T : rT;
                    kf = R.A;
#pragma unroll 1
                    for (int m = 0; m < abs(R.pw); ++m) kf *= b;
                } else {
                    kf = gdtk_exp(fma(R.mC, rT, fma(R.n, lnT, R.lnA)), tab.ETAB);
                }
                // P = (R T / P_atm)^sum(nu) prod E^nu from its first factor on
                double P = R.nusum > 0 ? cf : rcf;
                bool one = R.nusum == 0;   // no factor yet
                for (int m = 1; m < abs(R.nusum); ++m) P *= R.nusum > 0 ? cf : rcf;
                for (int k = 0; k < R.np; ++k) {
                    const int nk = R.anu[k];
                    const double v = (nk > 0 ? E : E + GDTK_NSP)[R.sp[k]];
                    int m = abs(nk);
                    if (one) { P = v; one = false; --m; }
                    for (; m > 0; --m) P *= v;
                }
                kb = one ? kf : kf * P;
            } else
#endif
            {
                double dg = 0.0;
                for (int k = 0; k < R.np; ++k) dg = fma(__hiloint2double(R.nuh[k], 0), G[R.sp[k]], dg);
                const double lnKc = fma(__hiloint2double(R.nusumh, 0), GDTK_LN_PATM_R - lnT, -dg);
                if (R.mode != 2) {
                    const double lkf = fma(R.mC, rT, fma(R.n, lnT, R.lnA));
                    kf = gdtk_exp(lkf, tab.ETAB);
                    kb = R.mode == 0 ? gdtk_exp(lkf - lnKc, tab.ETAB)
                                     : gdtk_exp(fma(R.mCb, rT, fma(R.nb, lnT, R.lnAb)), tab.ETAB);
                } else {
                    const double lkb = fma(R.mCb, rT, fma(R.nb, lnT, R.lnAb));
                    kb = gdtk_exp(lkb, tab.ETAB);
                    kf = gdtk_exp(lkb + lnKc, tab.ETAB);
                }
            }
            K[R.idx] = kf;
            K[GDTK_NR + R.idx] = kb;
        }
#if GDTK_NFALLOFF
#pragma unroll 1
        for (int f = gl; f < GDTK_NFALLOFF; f += L) {
            double kf, kb;
            falloff_rates(GDTK_FALL_TAB[f], T, lnT, rT, G[GDTK_NSP + f], G, 1, tab.ETAB, kf, kb);
            K[GDTK_FALL_TAB[f].idx] = kf;
            K[GDTK_NR + GDTK_FALL_TAB[f].idx] = kb;
        }
#endif
    }
    __syncwarp(GRP_FULL);
}

__device__ __forceinline__ double grp_ipow(double x, int n) {   // the order of ipow_expr (codegen.cpp)
    if (n == 1) return x;
    if (n == 2) return x * x;
    double p = 0.0, v = x;
    bool got = false;
    for (int m = n;;) {
        if (m & 1) { p = got ? p * v : v; got = true; }
        m >>= 1;
        if (!m) return p;
        v = v * v;
    }
}

#if GDTK_METHOD != 0
// The q and L sums of the alpha-QSS right-hand side on the integer pipe: a term takes about 22 cycles there, where
// an FP64 addition takes 76 of the pipe that bounds the kernel (74% busy with 65,536 cells), and the
// terms do not wait for one another.  The terms, all >= 0, are aligned to the largest with 5 bits below its last
// and the sum is rounded once, closer to the exact value than the chain of FP64 additions it replaces.  64 bits hold 64
// terms of the largest one's size; a longer sum (128 reactions can give one 384 entries) is that chain.
// 262,147 H2-air cells 400 -> 364 ms, 32,000 with 16 lanes 80.7 -> 72.0.  The tick rates' products stay FP64:
// on the integer pipe, with its conversions, they took 391 to 517 ms.
// sum of the entries' W 2^shift (index | shift << 16)
__device__ __forceinline__ double grp_gather(const unsigned* ent, int e0, int e1, const double* W) {
    const unsigned* H = reinterpret_cast<const unsigned*>(W) + 1;
    unsigned mx = 0, any = 0;
#pragma unroll 4
    for (int e = e0; e < e1; ++e) {
        const unsigned x = ent[e], h = H[2 * (x & 0xffff)];
        mx = max(mx, h + ((x >> 16) << 20));
        any |= h;
    }
    // at most 64 entries, no sign (the scaling carries that of -inf or a NaN out of mx), and a normal largest term, so
    // far from the range's ends that 64 of it have no infinite sum
    if (e1 - e0 <= 64 && (int)any >= 0 && mx - 0x03600000u < 0x7f800000u - 0x03600000u) {
        const int E6 = (int)(mx >> 20) + 6;   // the largest term's leading bit at 2^57
        uint64_t acc = 0;
#pragma unroll 4
        for (int e = e0; e < e1; ++e) {
            const unsigned x = ent[e];
            const uint64_t w = (uint64_t)dbits(W[x & 0xffff]);
            const int we = (int)(w >> 52), d = E6 - we - (int)(x >> 16);
            if (we != 0 && d < 64) acc += ((w << 11) | 0x8000000000000000ull) >> d;
        }
        const int c = __clzll((long long)acc);   // 0..6
        acc <<= c;
        return __longlong_as_double((long long)((acc >> 11) + ((acc >> 10) & 1) + ((uint64_t)(unsigned)(E6 - c - 1) << 52)));
    }
    double sum = 0.0;
    for (int e = e0; e < e1; ++e) {
        const unsigned x = ent[e];
        sum = fma((double)(1u << (x >> 16)), W[x & 0xffff], sum);
    }
    return sum;
}
#endif

// A third-body sum by G lanes (gl: the lane among them), in every lane: pairs of species with the second product fused, then
// grp_sum's tree.  With one species to a lane both lanes of a pair form it.
template <int G>
__device__ __forceinline__ double third_body_sum(int gl, const double* ef, const double* c) {
    constexpr int W = G < GRP_P2 ? G : GRP_P2, KC = GRP_P2 / W, KP = KC < 2 ? 1 : KC / 2;
    const int base = (gl & (W - 1)) * KC & ~1;
    double v[KP];
#pragma unroll
    for (int k = 0; k < KP; ++k) {
        const int i = base + 2 * k;
        v[k] = i < GDTK_NSP ? third_body(ef[i], c[i]) : 0.0;
        if (i + 1 < GDTK_NSP) v[k] = fma(ef[i + 1], c[i + 1], v[k]);
    }
#pragma unroll
    for (int w = 1; w < KP; w <<= 1)
#pragma unroll
        for (int k = 0; k < KP; k += 2 * w) v[k] += v[k + w];
#pragma unroll
    for (int x = KC < 2 ? 2 : 1; x < W; x <<= 1) v[0] += __shfl_xor_sync(GRP_FULL, v[0], x);
    return v[0];
}

// Lanes to a third-body sum: the L / G sums of a turn share its instructions, of which a sum takes P2 / G for its pairs,
// P2 / 2 G - 1 for its tree in a lane and log2 G over its lanes.  The G of the fewest FP64 instructions; 3 sets of Park's 5
// species with 32 lanes: 4 instructions where one sum after the other took 12 (4,096 cells 2.40 -> 2.04 ms).
constexpr int set_cost(int L, int G) {
    int lg = 0;
    for (int x = 1; x < G; x <<= 1) ++lg;
    return (GDTK_NSETS + L / G - 1) / (L / G) * (GRP_P2 / G < 2 ? 1 + lg : GRP_P2 / G + GRP_P2 / (2 * G) - 1 + lg);
}
constexpr int set_lanes(int L) {
    int best = L < GRP_P2 ? L : GRP_P2;
    for (int G = best; G >= 1 && GRP_P2 / G <= 4; G >>= 1)   // at most 4 values in a lane
        if (set_cost(L, G) < set_cost(L, best)) best = G;
    return best;
}

// q and L of every species at the concentrations c into S[GO_Q..], S[GO_L..] (gen_rhs).
template <int L>
__device__ __forceinline__ void grp_rhs(const GrpTab& tab, const GrpCell& s, const double* c, int gl, bool act) {
    double* S = s.S;
    constexpr int G = set_lanes(L);
    if (G == L) {   // one sum after the other
#pragma unroll 1
        for (int m = 0; m < GDTK_NSETS; ++m) {
            const double* ef = tab.eff + m * GDTK_NSP;
            const double M = third_body_sum<L>(gl, ef, c);
            if (act && gl == 0) S[GO_M + m] = M;
        }
    } else {
#pragma unroll 1
        for (int m0 = 0; m0 < GDTK_NSETS; m0 += L / G) {
            const int m = m0 + gl / G;
            const double M = third_body_sum<G>(gl & (G - 1), tab.eff + (m < GDTK_NSETS ? m : 0) * GDTK_NSP, c);
            if (act && m < GDTK_NSETS && !(gl & (G - 1))) S[GO_M + m] = M;
        }
    }
    __syncwarp(GRP_FULL);
    const double* K = S + GO_K;
    double* W = S + GO_W;
    if (act) {
#pragma unroll 1
        for (int r = gl; r < GDTK_NR; r += L) {
            const uint4 x = tab.rx[r];
            const int id = x.w & 0xffff, set = x.w >> 16;
            double wf = K[id], wb = K[GDTK_NR + id];
            const unsigned nf = x.z & 7, nb = (x.z >> 3) & 7;
            if (set) { const double M = S[GO_M + set - 1]; wf *= M; wb *= M; }
            unsigned sp = x.x, co = x.z >> 6;
            for (unsigned k = 0; k < nf; ++k, sp >>= 8, co >>= 3) wf *= grp_ipow(c[sp & 255], co & 7);
            sp = x.y; co = x.z >> 18;
            for (unsigned k = 0; k < nb; ++k, sp >>= 8, co >>= 3) wb *= grp_ipow(c[sp & 255], co & 7);
            W[id] = wf;
            W[GDTK_NR + id] = wb;
        }
    }
    __syncwarp(GRP_FULL);
    if (act) {
        constexpr int LV = L == 4 ? 0 : L == 8 ? 1 : L == 16 ? 2 : 3;
        const int* ls = tab.lane_start + 33 * LV;
        const int* lt = tab.lane_task + 2 * GDTK_NSP * LV;
#pragma unroll 1
        for (int k = ls[gl]; k < ls[gl + 1]; ++k) {
            const int t = lt[k], e1 = tab.task[t + 1];
#if GDTK_METHOD == 0
            int e = tab.task[t];
            double acc = 0.0;
            if (e < e1) {   // the first term: no sum, and no product by a coefficient of 1
                const unsigned x = tab.ent[e++];
                acc = W[x & 0xffff];
                if (x >> 16 != 1) acc *= __hiloint2double(GRP_COEF_HI[x >> 16], 0);
            }
#pragma unroll 4
            for (; e < e1; ++e) {
                const unsigned x = tab.ent[e];
                acc = fma(__hiloint2double(GRP_COEF_HI[x >> 16], 0), W[x & 0xffff], acc);
            }
#else
            const double acc = grp_gather(tab.ent, tab.task[t], e1, W);
#endif
            S[((t & 1) ? GO_L : GO_Q) + (t >> 1)] = acc;
        }
    }
    __syncwarp(GRP_FULL);
}

#if GDTK_MIX_THERMO
// mix_coeffs with the 8 sums over the lanes
template <int L>
__device__ __forceinline__ void grp_mix_coeffs(const double* TH, const double* YR, int seg, double* m, int gl, bool act) {
    if (act) {
#pragma unroll 1
        for (int k = gl; k < 8; k += L) {
            const double* c = TH + GDTK_TH_SEG0 + 24 * seg + k;
            double acc = 0.0;
#pragma unroll
            for (int i = 0; i < GDTK_NSP; ++i) acc = fma(YR[i], c[i * GDTK_TH_STRIDE], acc);
            m[k] = acc;
            if (k >= 3 && k < 7) m[5 + k] = __hiloint2double(k == 3 ? 0x40000000 : k == 4 ? 0x40080000 : k == 5 ? 0x40100000 : 0x40140000, 0) * acc;
        }
    }
    __syncwarp(GRP_FULL);
}
#endif

#if GDTK_MIX_THERMO
// mix_H_Cp's H/R (odd false) or Cp/R (odd true), each in its own roundings: Cp/R starts from 0 T + c
__device__ __forceinline__ double mix_H_or_Cp(const double* m, bool odd, double T, double lnT, double rT, double rT2) {
    const double a6 = odd ? 0.0 : m[6], a5 = m[odd ? 11 : 5], a4 = m[odd ? 10 : 4], a3 = m[odd ? 9 : 3], a2 = m[odd ? 8 : 2];
    const double h0 = odd ? -m[0] : m[0], e = m[odd ? 2 : 7];
    return fma(T, fma(T, fma(T, fma(T, fma(T, a6, a5), a4), a3), a2), fma(h0, odd ? rT2 : rT, fma(m[1], odd ? rT : lnT, e)));
}
#endif

// T_from_u for the groups with `act`; YR and the scratch M (24 doubles or 2 NSP) in the cell's slice.
template <int L>
__device__ __forceinline__ double grp_T_from_u(const GrpTab& tab, const double* YR, double* M, double u_tgt, double T_guess,
                                               double ysum, double& lnT_io, int& err, int& iters, int gl, bool act) {
    double T = T_guess, dT = 0.0, lnT = lnT_io, rT = 0.0;
    if (act) rT = gdtk_rcp(T);
    bool on = act;
#if GDTK_MIX_THERMO
    int seg_a = -1, seg_b = -1;
#endif
#pragma unroll 1
    for (int it = 0; it <= 10; ++it) {
        if (on && it > 0) {
            if (newton_advance(T, lnT, rT, dT)) on = false;
            else if (it == 10) { on = false; if (gt_pos(abs_bits(dT), 1e-3)) err = ST_NEWTON; }
        }
        if (!__any_sync(GRP_FULL, on)) break;
        const double rT2 = rT * rT;
        double f = 0.0, cv = 0.0;
#if GDTK_MIX_THERMO
        int sa = 0, sb = 0;
        double wb = 0.0;
        const bool mix = on && in_mix_range(T) && seg_of(tab.TH, T, sa, sb, wb);
        const bool na = mix && sa != seg_a, nb = mix && nonzero(wb) && sb != seg_b;
        if (__any_sync(GRP_FULL, na)) grp_mix_coeffs<L>(tab.TH, YR, sa, M, gl, na);
        if (__any_sync(GRP_FULL, nb)) grp_mix_coeffs<L>(tab.TH, YR, sb, M + 12, gl, nb);
        if (na) seg_a = sa;
        if (nb) seg_b = sb;
        if (__any_sync(GRP_FULL, mix)) {
            // H/R on the even lanes and Cp/R on the odd ones: the same polynomial in T with other coefficients
            const bool odd = gl & 1;
            double v = 0.0;
            if (mix) {
                v = mix_H_or_Cp(M, odd, T, lnT, rT, rT2);
                if (nonzero(wb)) v = fma(wb, mix_H_or_Cp(M + 12, odd, T, lnT, rT, rT2) - v, v);
                v = fma(-ysum, odd ? 1.0 : T, v);
            }
            const double o = __shfl_xor_sync(GRP_FULL, v, 1);
            f = odd ? o : v;
            cv = odd ? v : o;
        }
        const bool each = on && !mix;
#else
        const bool each = on;
#endif
        if (__any_sync(GRP_FULL, each)) {   // species by species, over the lanes, into the scratch
            int e = 0;
            if (each)
                for (int i = gl; i < GDTK_NSP; i += L) {
                    double tf, tc;
                    species_terms(tab.TH, i, YR[i], T, lnT, rT, rT2, tf, tc, e);
                    M[i] = tf;
                    M[GDTK_NSP + i] = tc;
                }
            __syncwarp(GRP_FULL);
            const double sf = grp_sum<L>(gl, [&](int i) { return M[i]; });
            const double sc = grp_sum<L>(gl, [&](int i) { return M[GDTK_NSP + i]; });
#pragma unroll
            for (int x = 1; x < L; x <<= 1) e |= __shfl_xor_sync(GRP_FULL, e, x);
            if (each) {
                f = sf;
                cv = sc;
                if (e) err = e;
            }
#if GDTK_MIX_THERMO
            if (each) seg_a = seg_b = -1;   // the coefficients are overwritten
#endif
        }
        if (on) { dT = -gdtk_div(f - u_tgt, cv); ++iters; }
    }
    __syncwarp(GRP_FULL);
    if (act) lnT_io = lnT;
    return T;
}

// One warp's loop with L lanes per cell.  Returns true when cells are left for twice the lanes.
template <int L>
__device__ __forceinline__ bool grp_loop(const FastArgs& a, const GrpTab& tab, GrpCell& s, bool& exhausted, bool first) {
    const int lane = threadIdx.x & 31, gl = lane & (L - 1), leader0 = lane & ~(L - 1);
    const unsigned gmask = (L == 32 ? GRP_FULL : ((1u << (L & 31)) - 1u)) << leader0;
    while (true) {
        if (!exhausted) {
            const unsigned need = __ballot_sync(GRP_FULL, !s.have && gl == 0);
            if (need) {
                // The first cells are dealt over the SMs, then the warps, then a warp's groups, so that the longest
                // lie in different SMs and warps and take a warp's lanes when its shorter ones are done; the
                // rest come from the counter, at most one atomic per warp.
                const unsigned warps = gridDim.x * (blockDim.x >> 5), dealt = warps * (32 / L);
                unsigned pos, next;
                if (first) {
                    pos = (lane / L) * warps + (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
                    next = dealt;
                    first = false;
                } else {
                    unsigned base = 0;
                    if (lane == 0) base = atomicAdd(a.counter, (unsigned)__popc(need));
                    base = dealt + __shfl_sync(GRP_FULL, base, 0);
                    pos = base + __popc(need & ((1u << leader0) - 1u));
                    next = base + __popc(need);
                }
                if (!s.have && pos < (unsigned)a.total) {
                    s.g = a.order ? (unsigned)a.order[pos] : pos;
                    int lo = 0, hi = a.nblocks - 1;
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) >> 1;
                        if ((unsigned)a.blocks[mid].first <= s.g) lo = mid; else hi = mid - 1;
                    }
                    s.b = lo;
                    const CellBlock& B = a.blocks[lo];
                    const int ci = (int)(s.g - (unsigned)B.first);
                    s.ci = ci;
                    s.rho = B.rho[ci]; s.u = B.u[ci]; s.tI = B.t_interval; s.dtS0 = B.dt_chem[ci];
                    if (B.T[ci] <= a.T_frozen) {
                        if (B.status && gl == 0) B.status[ci] = ST_FROZEN;
                    } else if (isnan(s.rho) || s.rho <= 0.0) {
                        if (B.status && gl == 0) B.status[ci] = ST_BAD;
                    } else {
                        s.have = true;
                        s.retried = false;
                        s.rrho = gdtk_rcp(s.rho);
                        s.n_steps = s.n_rhs = s.n_kc = s.n_newton = s.n_rej = s.n_est = 0;
                        s.phase = -1;
                    }
                }
                exhausted = next >= (unsigned)a.total;
            }
        }
        const unsigned hm = __ballot_sync(GRP_FULL, s.have);
        if (!hm) {
            if (exhausted) return false;
            continue;
        }
        if (L < 32 && exhausted && __popc(hm) <= 16) return true;

        double* const S = s.S;
        double* const Y0 = S + GO_Y0;
        double* const C = S + GO_C;
        double* const Q = S + GO_Q;
        double* const LO = S + GO_L;
        double* const W = S + GO_W;
        double* const V = S + GO_V;
        // as in gdtk_chem_fast, the third bodies of pressure-dependent rates see the input's concentrations unclipped
        const bool start = s.have && s.phase == -1, fresh = GDTK_NFALLOFF && start;
        if (__any_sync(GRP_FULL, start)) {   // (re)start from the stored input state
            if (start) {
                const CellBlock& B = a.blocks[s.b];
                s.T = B.T[s.ci]; s.p = B.p[s.ci]; s.dtS = s.dtS0; s.t = 0.0; s.err = 0;
                s.lnT = gdtk_log(s.T);
                for (int i = gl; i < GDTK_NSP; i += L) {
                    const double v = B.massf[(size_t)i * B.ncell + s.ci] * s.rho * GDTK_RM[i];
                    Y0[i] = (!GDTK_NFALLOFF && v < MIN_MOLES) ? 0.0 : v;
                }
                s.need_kc = true;
                s.phase = 0;
            }
            __syncwarp(GRP_FULL);
        }
        {
            const bool k = s.have && s.need_kc;
            if (__any_sync(GRP_FULL, k)) {
                grp_rate_constants<L>(tab, s, gl, k);
                if (k) { ++s.n_kc; s.need_kc = false; }
            }
            if (GDTK_NFALLOFF && __any_sync(GRP_FULL, fresh)) {
                if (fresh)
                    for (int i = gl; i < GDTK_NSP; i += L) Y0[i] = (Y0[i] < MIN_MOLES) ? 0.0 : Y0[i];
                __syncwarp(GRP_FULL);
            }
        }
        const bool act = s.have;
        if (act) ++s.n_steps;
        bool ok = false;

        // the first step size of a cell or subcycle, from the right-hand side at Y0 (in Q, LO)
        auto first_rhs = [&]() {
            double md = 1.0e6;
            const bool est = act && s.phase == 0 && !(s.dtS > s.tI) && s.dtS <= 0.0;
            if (__any_sync(GRP_FULL, est)) {
                if (est)
                    for (int i = gl; i < GDTK_NSP; i += L) md = estimate_of(Y0[i], Q[i], LO[i], md);
#pragma unroll
                for (int x = 1; x < L; x <<= 1) md = fmin(md, __shfl_xor_sync(GRP_FULL, md, x));
            }
            if (act && s.phase == 0) {
                if (s.dtS > s.tI) s.h = s.tI;
                else if (s.dtS <= 0.0) { s.h = estimate_clip(md); ++s.n_est; ++s.n_rhs; }
                else s.h = s.dtS;
                s.cycle = 0;
                s.phase = 1;
            }
            if (act && s.phase == 1) {
                s.dtSave = s.dtS;
                const double left = s.tI - s.t;
                s.h = lt_pos(s.h, left) ? s.h : left;
                s.attempt = 0;
                s.phase = 2;
            }
        };
#if GDTK_METHOD == 0
#pragma unroll 1
        for (int st = 0; st < 6; ++st) {
            grp_rhs<L>(tab, s, st == 0 ? Y0 : C, gl, act);
            if (act) ++s.n_rhs;
            if (st == 0) first_rhs();
            double* kv = V + st * GDTK_NSP;
            if (act) {
#pragma unroll 1
                for (int i = gl; i < GDTK_NSP; i += L) {
                    kv[i] = Q[i] - LO[i];
                    if (st < 5) {
                        double acc = RKF_A[st][0] * V[i];
                        for (int j = 1; j <= st; ++j) acc = fma(RKF_A[st][j], V[j * GDTK_NSP + i], acc);
                        C[i] = fma(s.h, acc, Y0[i]);
                    } else {
                        double o, e;
                        rkf_result(V[i], V[2 * GDTK_NSP + i], V[3 * GDTK_NSP + i], V[4 * GDTK_NSP + i], V[5 * GDTK_NSP + i],
                                   s.h, Y0[i], o, e);
                        C[i] = o;
                        W[i] = __dmul_rn(e, e);
                    }
                }
            }
            __syncwarp(GRP_FULL);
        }
        {
            const double err2 = grp_sum<L>(gl, [&](int i) { return W[i]; });
            if (act) s.dtS = rkf_scale(err2 * (1.0 / GDTK_NSP), tab.ETAB, ok) * s.h;
        }
#else
        {
            double* const Q0 = V;
            double* const P0 = V + GDTK_NSP;
            double* const YP0 = V + 2 * GDTK_NSP;
            bool open = act, conv = false;
#pragma unroll 1
            for (int st = 0; st <= GDTK_MAX_ITERS; ++st) {
                grp_rhs<L>(tab, s, st == 0 ? Y0 : C, gl, open);
                if (open) ++s.n_rhs;
                if (st == 0) first_rhs();
                bool cv = true;
                if (open) {
#pragma unroll 1
                    for (int i = gl; i < GDTK_NSP; i += L) {
                        const double y = Y0[i], q = Q[i];
                        double v;
                        if (st == 0) {
                            const double pp = qss_p(LO[i], y);
                            v = qss_predict(y, pp, s.h, q);
                            Q0[i] = q;
                            P0[i] = half_nn(pp);
                            YP0[i] = v;
                        } else {
                            const double pp = qss_p(LO[i], C[i]);
                            v = qss_value(y, pp, s.h, q, Q0[i], fma(0.5, pp, P0[i]));
                            if (qss_misses(v, YP0[i])) cv = false;
                        }
                        C[i] = v;
                    }
                }
                const unsigned miss = __ballot_sync(GRP_FULL, open && !cv);
                if (open && st > 0 && !(miss & gmask)) { conv = true; open = false; }
                __syncwarp(GRP_FULL);
                if (!__any_sync(GRP_FULL, open)) break;
            }
            const Ratio sg = grp_max_ratio<L>(gl, [&](int i) { return sigma_leaf(C[i], YP0[i]); });
            if (act) s.dtS = qss_step(sg, s.h);
            ok = conv;
        }
#endif
        // mass-fraction test (chemistry_update.d:175-185); the Y_i go to W for the thermo update
        if (act)
            for (int i = gl; i < GDTK_NSP; i += L) W[i] = clipped_massf(C[i], GDTK_M[i], s.rrho);
        __syncwarp(GRP_FULL);
        const double tot = grp_sum<L>(gl, [&](int i) { return W[i]; });
        if (gt_pos(abs_bits(tot - 1.0), ALLOWABLE_MASSF_ERROR)) ok = false;
        ok = ok && act;
        int fail = 0;
        bool done = false;
        if (ok) {
            s.t += s.h;
            for (int i = gl; i < GDTK_NSP; i += L) Y0[i] = C[i];
            s.h = grown_step(s.h, s.dtS);
        }
#if GDTK_TIGHT
        if (__any_sync(GRP_FULL, ok)) {
            if (ok)
                for (int i = gl; i < GDTK_NSP; i += L) W[i] = __dmul_rn(W[i], GDTK_R[i]);
            __syncwarp(GRP_FULL);
            const double Rm = grp_sum<L>(gl, [&](int i) { return W[i]; });
            const double Tn = grp_T_from_u<L>(tab, W, W + GDTK_NSP, s.u, s.T, Rm, s.lnT, s.err, s.n_newton, gl, ok);
            if (ok) {
                s.T = Tn;
                s.p = s.rho * Rm * Tn;
                s.need_kc = true;
            }
        }
#endif
        if (ok) {
            if (s.err) fail = s.err;
            else if (ge_pos(s.t, s.tI)) {
                if (s.cycle == 0) s.dtSave = s.dtS;
                done = true;
            } else {
                ++s.cycle;
                if (s.cycle == GDTK_MAX_SUBCYCLES) fail = ST_MAX_SUBCYCLES;
                else s.phase = 1;
            }
        } else if (act) {
            ++s.n_rej;
            s.h = gdtk_div(s.h, 10.0);
            if (s.err) fail = s.err;
            else if (s.h < H_MIN) fail = ST_H_MIN;
            else if (++s.attempt == GDTK_MAX_ATTEMPTS) fail = ST_MAX_ATTEMPTS;
        }
        if (fail) {
            const bool retryable = fail == ST_H_MIN || fail == ST_MAX_ATTEMPTS || fail == ST_MAX_SUBCYCLES;
            if ((a.flags & F_RETRY) && retryable && !s.retried) {   // fluidfvcell.d:924-941
                s.retried = true;
                s.dtS0 = -1.0;
                s.phase = -1;
            } else {
                if (a.blocks[s.b].status && gl == 0) a.blocks[s.b].status[s.ci] = fail;
                s.have = false;
            }
        }
        __syncwarp(GRP_FULL);
        if (__any_sync(GRP_FULL, done)) {   // chemistry_update.d:290-325, then fluidfvcell.d:956
            if (done)
                for (int i = gl; i < GDTK_NSP; i += L) W[i] = clipped_massf(Y0[i], GDTK_M[i], s.rrho);
            __syncwarp(GRP_FULL);
            double rtot = grp_sum<L>(gl, [&](int i) { return W[i]; });
            if (done) rtot = gdtk_rcp(rtot);
            __syncwarp(GRP_FULL);
            if (done)
                for (int i = gl; i < GDTK_NSP; i += L) {
                    const double y = W[i] * rtot;
                    C[i] = y;
                    W[i] = __dmul_rn(y, GDTK_R[i]);
                }
            __syncwarp(GRP_FULL);
            int st = 0;
            if (a.flags & F_UPDATE_THERMO) {
                const double Rm = grp_sum<L>(gl, [&](int i) { return W[i]; });
                const double Tn = grp_T_from_u<L>(tab, W, W + GDTK_NSP, s.u, s.T, Rm, s.lnT, st, s.n_newton, gl, done);
                if (done) {
                    s.T = Tn;
                    s.p = s.rho * Rm * Tn;
                }
            }
            if (done) {
                const CellBlock& B = a.blocks[s.b];
                if (!st) {
                    for (int i = gl; i < GDTK_NSP; i += L) B.massf[(size_t)i * B.ncell + s.ci] = C[i];
                    if (gl == 0) {
                        B.T[s.ci] = s.T;
                        B.p[s.ci] = s.p;
                        B.dt_chem[s.ci] = s.dtSave;
                    }
                }
                if (B.status && gl == 0) B.status[s.ci] = st;
                s.have = false;
            }
        }
        if (act && !s.have && gl == 0) {
            if (a.cell_counters) {
                const size_t n = (size_t)a.total;
                a.cell_counters[0 * n + s.g] = s.n_steps;
                a.cell_counters[1 * n + s.g] = s.n_rhs;
                a.cell_counters[2 * n + s.g] = s.n_kc;
                a.cell_counters[3 * n + s.g] = s.n_newton;
                a.cell_counters[4 * n + s.g] = s.n_rej;
                a.cell_counters[5 * n + s.g] = s.n_est;
            }
            if (a.totals) {
                atomicAdd(a.totals + 0, (unsigned long long)s.n_steps);
                atomicAdd(a.totals + 1, (unsigned long long)s.n_rhs);
                atomicAdd(a.totals + 2, (unsigned long long)s.n_kc);
                atomicAdd(a.totals + 3, (unsigned long long)s.n_newton);
                atomicAdd(a.totals + 4, (unsigned long long)s.n_rej);
                atomicAdd(a.totals + 5, (unsigned long long)s.n_est);
            }
        }
        __syncwarp(GRP_FULL);
    }
}

// The cells left by groups of L lanes, handed to groups of 2 L: at most 16 / L of them.
template <int L>
__device__ __forceinline__ void grp_widen(GrpCell& s) {
    const unsigned hm = __ballot_sync(GRP_FULL, s.have && (threadIdx.x & (L - 1)) == 0);   // leaders that hold a cell
    int k = (threadIdx.x & 31) / (2 * L);
    unsigned m = hm;
    while (k-- > 0) m &= m - 1;
    const int src = m ? __ffs(m) - 1 : (threadIdx.x & 31);
    const bool have = m != 0;
    auto mv = [&](auto& v) { v = __shfl_sync(GRP_FULL, v, src); };
    unsigned long long p = __shfl_sync(GRP_FULL, (unsigned long long)s.S, src);
    // a group without a cell keeps some slice that no cell uses: it writes nothing
    s.S = (double*)p;
    mv(s.g); mv(s.b); mv(s.ci); mv(s.phase); mv(s.cycle); mv(s.attempt); mv(s.err);
    int r = __shfl_sync(GRP_FULL, (int)s.retried, src), kc = __shfl_sync(GRP_FULL, (int)s.need_kc, src);
    s.retried = r; s.need_kc = kc;
    mv(s.rho); mv(s.rrho); mv(s.u); mv(s.T); mv(s.lnT); mv(s.p); mv(s.dtS); mv(s.dtS0); mv(s.dtSave); mv(s.h); mv(s.t); mv(s.tI);
    mv(s.n_steps); mv(s.n_rhs); mv(s.n_kc); mv(s.n_newton); mv(s.n_rej); mv(s.n_est);
    s.have = have;
    __syncwarp(GRP_FULL);
}

extern "C" __global__ void __launch_bounds__(GDTK_GRP_BLOCK) gdtk_chem_group(const __grid_constant__ FastArgs a, int lanes) {
    extern __shared__ double smem[];
    GrpTab tab;
    double* q = smem;
    auto stage = [&](const void* from, size_t bytes) {   // whole doubles
        const double* f = (const double*)from;
        const int n = (int)((bytes + 7) / 8);
        for (int k = threadIdx.x; k < n; k += blockDim.x) q[k] = f[k];
        double* at = q;
        q += n;
        return (const void*)at;
    };
    tab.rx = (const uint4*)stage(GRP_RX, sizeof GRP_RX);     // first: 16-byte aligned
    tab.TH = (const double*)stage(a.thermo, (size_t)GDTK_NSP * GDTK_TH_STRIDE * 8);
    tab.ETAB = (const uint64_t*)stage(a.exp_table, GDTK_EXP2_TABLE_SIZE * 8);
    tab.eff = (const double*)stage(GRP_EFF, sizeof GRP_EFF);
    tab.kc = (const GrpKc*)stage(GRP_KC, sizeof GRP_KC);
    tab.ent = (const unsigned*)stage(GRP_ENT, sizeof GRP_ENT);
    tab.task = (const int*)stage(GRP_TASK, sizeof GRP_TASK);
    tab.lane_start = (const int*)stage(GRP_LANE_START, sizeof GRP_LANE_START);
    tab.lane_task = (const int*)stage(GRP_LANE_TASK, sizeof GRP_LANE_TASK);
    __syncthreads();
    GrpCell s{};
    const int cells = 32 / lanes;   // of a warp
    s.S = q + ((threadIdx.x >> 5) * cells + (threadIdx.x & 31) / lanes) * GRP_CELL;
    bool exhausted = false, left = true;
    if (lanes == 4) { left = grp_loop<4>(a, tab, s, exhausted, true); if (left) grp_widen<4>(s); }
    if (lanes <= 8 && left) { left = grp_loop<8>(a, tab, s, exhausted, lanes == 8); if (left) grp_widen<8>(s); }
    if (lanes <= 16 && left) { left = grp_loop<16>(a, tab, s, exhausted, lanes == 16); if (left) grp_widen<16>(s); }
    if (left) grp_loop<32>(a, tab, s, exhausted, lanes == 32);
}

}  // namespace gdtk_fast
#endif

// Device code shared by the move kernels (rmx_moves.cu) and the fused stage
// kernel (rmx_stage.cu): hashing, the code-length change of a candidate, the
// cached module terms.
#pragma once
#include <climits>

#include "rmx_engine.cuh"

// the total-exit term of every candidate through log1p of a per-unit log (1) or a log each (0)
#ifndef RMX_LOG1P
#define RMX_LOG1P 1
#endif

namespace rmx {

constexpr int32_t kEmpty = -1;
constexpr int32_t kNewMod = -2;

// ---------------------------------------------------------------- helpers

__device__ __forceinline__ uint32_t mix32(uint32_t x) {
    x ^= x >> 16;
    x *= 0x7feb352dU;
    x ^= x >> 15;
    x *= 0x846ca68bU;
    x ^= x >> 16;
    return x;
}

__device__ __forceinline__ int tab_slot(int32_t key, int mask) { return (int)(mix32((uint32_t)key) & (uint32_t)mask); }

__device__ __forceinline__ bool better(double d1, int32_t m1, double d2, int32_t m2) {
    return d1 < d2 || (d1 == d2 && m1 < m2);
}

// Everything about the moving unit that every candidate needs. The terms of
// the code-length change that depend only on the unit and its old module
// (Module.cpp:1109-1112: sumAllExitPr, exit and stay of the old module before
// and after) are folded into K once per unit.
struct UnitCtx {
    double pu, tu, eu, cu;  // flow, teleport weight, exit, tau*p + (1-tau)*d
    double eA, nexA;        // old module exit before / after the unit leaves
    double sum_exit;
    double K;               // -plogp(se) - 2 (plogp(nexA) - plogp(eA)) + plogp(nexA + nPA) - plogp(eA + PA)
    double S0, logS0, rS0;  // the new total exit without the target's change, its log and reciprocal
    int32_t A;
};

// plogp of the new total exit flow S0 + dm, where dm = (new - old exit of the
// target module) is tiny next to S0 for almost every candidate: then
// log(S0 + dm) = log(S0) + log1p(dm / S0) with log(S0) computed once per unit
// and log1p by its Mercator series through t^6 (|t| < 2^-10: truncation below
// 2^-70 / 7 of the value, far under FP64 rounding); otherwise the direct log.
__device__ __forceinline__ double plogp_total(const UnitCtx &c, double dm) {
#if RMX_LOG1P
    const double t = dm * c.rS0;
    if (c.rS0 > 0.0 && fabs(t) < 0x1p-10) {
        const double a = 1.0 - t * (0.5 - t * (1.0 / 3.0 - t * (0.25 - t * (0.2 - t * (1.0 / 6.0)))));
        return __dmul_rn(c.S0 + dm, __fma_rn(t, a, c.logS0));
    }
#endif
    return plogp(c.S0 + dm);
}

// Change of moving the unit into module with statistics st, given the unit's
// link flow to and from it (fixed point, out-links plus in-links, before the
// 1-tau factor): d_all - 2 d_exit + d_stay of Module.cpp:1109-1115 with the
// unit terms in K. The out- and in-flows (Module.cpp:1058, :1059) enter the
// change only through their sum (the new exit, :1104), so the tables keep one
// sum per module. t = the module's cached {plogp(exit), plogp(exit + P)}.
// pair(x, y) = {plogp(x), plogp(y)}.
template <typename Pair>
__device__ __forceinline__ double candidate_delta(const UnitCtx &c, const ModRec &r, fx_t sfx, Pair pair) {
    const double em = r.em;
    const double om_im = __fma_rn(r.g, c.tu, __fma_rn(kBeta, from_fx(sfx), __dmul_rn(c.cu, r.TW)));  // :1058 + :1059
    const double nexm = em + c.eu - om_im;                                 // Module.cpp:1104
    // new total exit sumAllExitPr + (nexA - eA) + (nexm - em), Module.cpp:1106
    const double2 p = pair(nexm, nexm + r.P + c.pu);
    return plogp_total(c, nexm - em) + c.K - 2.0 * (p.x - r.t.x) + (p.y - r.t.y);
}
__device__ __forceinline__ double candidate_delta(const UnitCtx &c, const ModRec &r, fx_t sfx) {
    return candidate_delta(c, r, sfx, [](double x, double y) { return make_double2(plogp(x), plogp(y)); });
}

// alpha p + beta d.
__device__ __forceinline__ double mix_flows(double p, double d) {
    return __fma_rn(kAlpha, p, __dmul_rn(kBeta, d));
}

// The hub pipeline's terms of a unit; its order of rounding the flow between the
// unit and its old module differs from the other bins' in the last bit.
__device__ __forceinline__ UnitCtx make_ctx(const Stat4 &ua, const ModRec &mA, double sum_exit, int32_t A,
                                            fx_t sA) {
    const double2 tA = mA.t;
    UnitCtx c;
    c.pu = from_fx(ua.P);
    c.tu = from_fx(ua.TW);
    const double du = from_fx(ua.D);
    c.eu = exit_flow(c.pu, c.tu, du, from_fx(ua.OUT));
    c.cu = mix_flows(c.pu, du);
    const double PA = mA.P, TWA = mA.TW, DA = mA.D;
    c.eA = mA.em;
    // outFlow + inFlow to the old module (Module.cpp:1047, :1048), sA = their link flows' sum
    const double fA = from_fx(sA), dT = TWA - c.tu;
    const double outA_inA = __fma_rn(mix_flows(PA - c.pu, DA - du), c.tu, __fma_rn(kBeta, fA, __dmul_rn(c.cu, dT)));
    c.nexA = c.eA - c.eu + outA_inA;  // :1084
    c.sum_exit = sum_exit;
    c.K = -plogp(sum_exit) - 2.0 * (plogp(c.nexA) - tA.x) + (plogp(c.nexA + (PA - c.pu)) - tA.y);
    c.S0 = sum_exit + c.nexA - c.eA;
#if RMX_LOG1P
    const bool pos = c.S0 > 0.0;
    c.logS0 = pos ? log(c.S0) : 0.0;
    c.rS0 = pos ? 1.0 / c.S0 : 0.0;
#else
    c.logS0 = c.rS0 = 0.0;
#endif
    c.A = A;
    return c;
}

__device__ __forceinline__ ModRec load_mod(const ModRec *p) {
    const double2 a = *reinterpret_cast<const double2 *>(&p->P), b = *reinterpret_cast<const double2 *>(&p->em);
    ModRec r;
    r.P = a.x;
    r.TW = a.y;
    r.em = b.x;
    r.g = b.y;
    r.t = p->t;
    return r;
}

__device__ __forceinline__ Stat4 load_stat(const Stat4 *p) {
    const longlong2 a = *reinterpret_cast<const longlong2 *>(&p->P);
    const longlong2 b = *reinterpret_cast<const longlong2 *>(&p->D);
    Stat4 r;
    r.P = a.x;
    r.TW = a.y;
    r.D = b.x;
    r.OUT = b.y;
    return r;
}

// A unit's terms by a group of W >= 8 lanes (gl = lane in the group): its six
// logarithms (old module before and after, total exit, and the two of the
// empty-module option, Module.cpp:1072-1077: exit e_u, no shared flow) are taken
// by six lanes in one call instead of one after another by all of them.
__device__ __forceinline__ UnitCtx make_ctx_lanes(int W, const Stat4 &ua, const ModRec &mA, double DA, double sum_exit, int32_t A,
                                                  fx_t sA, int gl, double &new_exit, double &new_stay) {
    const double2 tA = mA.t;
    UnitCtx c;
    c.pu = from_fx(ua.P);
    c.tu = from_fx(ua.TW);
    const double du = from_fx(ua.D);
    c.eu = exit_flow(c.pu, c.tu, du, from_fx(ua.OUT));
    c.cu = mix_flows(c.pu, du);
    const double PA = mA.P, TWA = mA.TW;
    c.eA = mA.em;
    const double outA_inA = __fma_rn(mix_flows(PA - c.pu, DA - du), c.tu,
                                     __fma_rn(c.cu, TWA - c.tu, __dmul_rn(kBeta, from_fx(sA))));
    c.nexA = c.eA - c.eu + outA_inA;
    c.sum_exit = sum_exit;
    c.S0 = sum_exit + c.nexA - c.eA;
    const double x = gl == 0   ? c.nexA
                     : gl == 1 ? c.nexA + (PA - c.pu)
                     : gl == 2 ? c.S0
                     : gl == 3 ? sum_exit
                     : gl == 4 ? c.eu
                               : c.eu + c.pu;
    const bool pos = x > 0.0;
    const double lg = pos ? log(x) : 0.0;
    const double pl = pos ? __dmul_rn(x, lg) : 0.0;
    const double p0 = __shfl_sync(0xffffffffu, pl, 0, W), p1 = __shfl_sync(0xffffffffu, pl, 1, W),
                 ps = __shfl_sync(0xffffffffu, pl, 3, W);
    c.logS0 = __shfl_sync(0xffffffffu, lg, 2, W);
    new_exit = __shfl_sync(0xffffffffu, pl, 4, W);
    new_stay = __shfl_sync(0xffffffffu, pl, 5, W);
    c.K = -ps - 2.0 * (p0 - tA.x) + (p1 - tA.y);
    c.rS0 = c.S0 > 0.0 ? 1.0 / c.S0 : 0.0;
    c.A = A;
    return c;
}

// Lowest (change, module) over the warp. The change as an order-preserving
// pair of 32-bit words, so that three hardware minimum reductions do it.
__device__ __forceinline__ void warp_best(double &d, int32_t &m) {
    const long long b = __double_as_longlong(d + 0.0);  // -0.0 counts as 0.0
    const unsigned long long o =
        b < 0 ? ~(unsigned long long)b : (unsigned long long)b ^ 0x8000000000000000ull;
    const unsigned h = (unsigned)(o >> 32), l = (unsigned)o;
    const unsigned mh = __reduce_min_sync(0xffffffffu, h);
    const unsigned ml = __reduce_min_sync(0xffffffffu, h == mh ? l : 0xffffffffu);
    m = __reduce_min_sync(0xffffffffu, h == mh && l == ml ? m : INT_MAX);
    const unsigned long long r = ((unsigned long long)mh << 32) | ml;
    d = __longlong_as_double(r & 0x8000000000000000ull ? (long long)(r ^ 0x8000000000000000ull) : (long long)~r);
}

__device__ __forceinline__ unsigned long long claim_key(uint32_t stamp, int32_t u) {
    return ((unsigned long long)stamp << 32) | (0xffffffffu - (uint32_t)u);
}

// A module's cached terms and its evaluation record.
__device__ __forceinline__ void write_terms(const Stat4 *mstat, double2 *term, ModRec *rec, int32_t m) {
    const Stat4 st = mstat[m];
    ModRec r;
    r.P = from_fx(st.P);
    r.TW = from_fx(st.TW);
    r.D = from_fx(st.D);
    r.em = exit_flow(r.P, r.TW, r.D, from_fx(st.OUT));
    r.g = mix_flows(r.P, r.D);
    r.t = make_double2(plogp(r.em), plogp(r.em + r.P));
    r.pad = 0.0;
    term[m] = r.t;
    rec[m] = r;
}

// Upper degree bounds of the warp, mid, block and large bins (run-time tuning).
struct BinBounds {
    int32_t warp, mid, block, large;
};

// degree bins: 8 / 16 / 32 lanes in registers, warp (shared table), block
// (shared table), hub (global table)
constexpr int kBins = 8;
constexpr int kBinReg8 = 0, kBinReg16 = 1, kBinReg32 = 2, kBinWarp = 3, kBinMid = 4, kBinBlock = 5, kBinLarge = 6,
              kBinHub = 7;

}  // namespace rmx

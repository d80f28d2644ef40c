// A whole stage of move sweeps as one cooperative launch.
//
// The sweeps of a stage (rmx_graph::stage_sweeps, and the coarse-tune
// sub-problems' loop) are short on most levels: a sub-batch of a few thousand
// units takes less time than the dozen dependent kernels that the pipeline of
// rmx_moves.cu needs for it. Here one persistent grid runs every sweep of the
// stage and its stop rule, with a grid barrier where that pipeline has a
// kernel boundary. Per sweep:
//   count    active units per (sub-batch, degree bin), empty modules per block
//   fill     a 32-byte record per active unit, grouped by (sub-batch, bin);
//            the ascending list of empty modules
//   per sub-batch
//     evaluate  every unit's best module; a proposer of an empty module bids
//               for one at once (the bid needs nothing of other units)
//     apply     movers' flow, teleport weight, dangling flow and out-flow move
//               between module statistics; unit memberships still read as they
//               were, a mover's target comes from its proposal
//     update    memberships, and the cached terms of the modules touched
//   length   code length from the module terms, stop rule
// Decisions, sums and bids are those of rmx_moves.cu (same arithmetic per
// candidate, exact integer sums, the same hashes), so partitions and code
// lengths are the same bit for bit.
//
// What bounds it: on levels of up to some 10^5 units the latency of a unit's
// chain (record, links, modules, table, module records, logarithms: 3 to 6 us)
// and the barriers (1.2 us each, three per sub-batch); beyond that the chain's
// latency over 16 warps per SM. One 512-thread block per SM with 128 registers:
// two blocks at 64 registers spilt the chain's values to local memory and took
// 431 against 379 us per sub-batch of the 1M-node planted graph's node level,
// and 10.8 against 6.5 us on a 44-unit level. Measured as whole runs against
// the kernel pipeline as it was then: 1000 nodes 2.78 -> 1.97 ms, 20,011 nodes in
// normal mode 19.0 -> 13.0 ms, 150,001 nodes 83 -> 64 ms. Levels of more than
// 2^23 links (unions: kFusedMaxUnionLinks in rmx_engine.cu) are left to that
// pipeline's kernels of 32 warps per SM.
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "rmx_moves.cuh"

namespace cg = cooperative_groups;

namespace rmx {
namespace {

constexpr unsigned kFull = 0xffffffffu;
// One 512-thread block per SM; its 8192 table slots serve one unit by 16 warps,
// four by 4 warps or 16 by a warp, each team using its own warps' slice.
constexpr int kSwT = 512, kSwWarps = kSwT / 32, kSwTab = 8192, kWarpTab = kSwTab / kSwWarps;
#ifndef RMX_STAGE_MINB
#define RMX_STAGE_MINB 1
#endif
constexpr int kWarpList = 256;  // slots a warp can have filled: 4096 links / 16 warps
constexpr int kMaxBuckets = 256, kMaxSub = 32;
constexpr int kIlp = 4;
constexpr size_t kStageSmem = (size_t)kSwTab * 12 + (size_t)kSwWarps * kWarpList * sizeof(uint16_t);

// An active unit of the sweep: its link ranges, its module (which only its own
// move changes, so it holds until its sub-batch is applied).
struct __align__(32) URec {
    uint32_t ob, ib;  // link offsets fit 32 bits: a graph has fewer than 2^31 links
    int32_t dout, din;
    int32_t u, A, pad0, pad1;
};

// Counters of a sweep, two sets used in turn (one is cleared while the other is in use).
struct SweepSet {
    unsigned cnt[kMaxBuckets], cur[kMaxBuckets];
    int any[kMaxSub];               // the sub-batch has a proposal
    unsigned next[kMaxSub][3];      // units taken of its light, mid and block, and large bins
    fx_t acc[3];                    // one instance: code-length sums
    unsigned long long remaining;   // instances still sweeping
};

struct StageDev {
    // level
    int32_t n;
    const int64_t *out_off, *in_off;
    const int32_t *out_dst, *in_src;
    const fx_t *out_fx, *in_fx;
    const Stat4 *attr;
    int32_t *mod;
    const int32_t *uinst;
    // modules, instances
    int32_t cap;
    Stat4 *stat;
    double2 *term;
    ModRec *rec;
    int32_t *mcount, *minst;
    int32_t K;
    double *sum_exit, *L;
    const fx_t *s0;
    fx_t *acc;
    uint8_t *active;
    // work
    URec *urec;
    int32_t *tgt;  // per record: the proposal (-1 none, -(m + 3) a bid for the empty module m)
    int32_t *prop;
    uint32_t *stamp;
    uint8_t *next_active;
    int32_t *free_list, *free_cnt;
    unsigned long long *claim;
    SweepSet *set;
    int64_t *ctl;  // [0] sweeps run
    // options
    int prior, allow_new, subtune, max_iter, nsub;
    double vthresh, threshold, ln2;
    uint32_t run_seed, stamp0;
    unsigned long long sweep0;
    BinBounds bb;
};

// The block's table in dynamic shared memory, by slot number: keys, and the
// slots' fixed-point sums in two halves (32-bit shared atomics are native, a
// 64-bit one is a loop of compare-and-swaps: 207 against 86 cycles of latency,
// a sixth of the throughput); then each warp's list of the slots it filled.
extern __shared__ __align__(16) unsigned char stage_smem[];
__device__ __forceinline__ int32_t &slot_key(int s) { return reinterpret_cast<int32_t *>(stage_smem)[s]; }
__device__ __forceinline__ unsigned &slot_lo(int s) { return reinterpret_cast<unsigned *>(stage_smem)[kSwTab + s]; }
__device__ __forceinline__ unsigned &slot_hi(int s) { return reinterpret_cast<unsigned *>(stage_smem)[2 * kSwTab + s]; }
__device__ __forceinline__ uint16_t &warp_list(int k) {
    return reinterpret_cast<uint16_t *>(stage_smem + (size_t)kSwTab * 12)[(threadIdx.x >> 5) * kWarpList + k];
}

// Barrier of a team of NW warps whose first warp is w0.
__device__ __forceinline__ int team_bar(int NW, int w0) { return NW == 16 ? 5 : 1 + (w0 >> 2); }
__device__ __forceinline__ void team_sync(int NW, int bar) {
    if (NW == 1)
        __syncwarp();
    else
        asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(NW * 32) : "memory");
}

__device__ __forceinline__ void add_slot(int s, fx_t q) {
    const unsigned ql = (unsigned)q, qh = (unsigned)((unsigned long long)q >> 32);
    const unsigned old = atomicAdd(&slot_lo(s), ql);
    atomicAdd(&slot_hi(s), qh + (old + ql < old ? 1u : 0u));
}

// Slot s's sum; the slot is emptied.
__device__ __forceinline__ fx_t take_slot(int s) {
    const fx_t v = (fx_t)(((unsigned long long)slot_hi(s) << 32) | slot_lo(s));
    slot_key(s) = kEmpty;
    slot_lo(s) = 0;
    slot_hi(s) = 0;
    return v;
}

__device__ __forceinline__ URec load_rec(const URec *p) {
    const int4 a = *reinterpret_cast<const int4 *>(&p->ob);
    const int2 b = *reinterpret_cast<const int2 *>(&p->u);
    URec r;
    r.ob = (uint32_t)a.x;
    r.ib = (uint32_t)a.y;
    r.dout = a.z;
    r.din = a.w;
    r.u = b.x;
    r.A = b.y;
    return r;
}

// Link j of a unit (out-links first): its place in the out or the in arrays.
__device__ __forceinline__ uint32_t link_at(const URec &r, int j, bool &isout) {
    isout = j < r.dout;
    return isout ? r.ob + (uint32_t)j : r.ib + (uint32_t)(j - r.dout);
}

// {plogp(x), plogp(y)} as one function of the kernel's: the logarithm's code and
// coefficients then exist once, not at every use, where they cost the registers
// and instruction-cache room of the loops around them.
__device__ __noinline__ double2 plogp2(double x, double y) { return make_double2(plogp(x), plogp(y)); }

// What one sub-batch's phases share.
struct SubCtx {
    uint32_t stamp, hseed;
    int64_t n_free;
    int *any;
    double sum_exit;  // one instance: its total exit
};

// The decision for record i from the best candidate (finish_unit of
// rmx_moves.cu), with the bid of k_claim. leader: the lane that writes it.
// Returns whether the unit found a move (it activates its neighbours).
__device__ __forceinline__ bool decide(const StageDev &a, const SubCtx &sc, int i, int32_t u, const UnitCtx &c, int32_t nA,
                                       double new_exit, double new_stay, double best, int32_t bm, bool leader) {
    if (a.allow_new && nA > 1) {
        const double dn = plogp_total(c, c.eu) + c.K - 2.0 * new_exit + new_stay;
        if (better(dn, INT_MAX, best, bm)) {
            best = dn;
            bm = kNewMod;
        }
    }
    const bool act = bm != INT_MAX && best < a.vthresh;
    if (leader) {
        int32_t out = -1;
        if (act) {
            out = bm;
            if (bm >= 0) {
                if (nA == 1 && a.mcount[bm] == 1 && bm > c.A) out = -1;
            } else {
                out = -1;
                if (sc.n_free > 0) {
                    int64_t s = mix32((uint32_t)u ^ sc.hseed) % sc.n_free;
                    for (int probe = 0; probe < 8; probe++, s = (s + 1) % sc.n_free) {
                        const int32_t m = a.free_list[s];
                        if (a.mcount[m] == 0) {
                            atomicMax(a.claim + m, claim_key(sc.stamp, u));
                            out = -(m + 3);
                            break;
                        }
                    }
                }
            }
            if (out != -1) {
                a.prop[u] = out;
                a.stamp[u] = sc.stamp;
                *sc.any = 1;
            }
        }
        a.tgt[i] = out;
    }
    return act;
}

__device__ __forceinline__ double unit_sum_exit(const StageDev &a, const SubCtx &sc, int32_t u) {
    return a.K == 1 ? sc.sum_exit : a.sum_exit[a.uinst[u]];
}

// Units of at most W = 8, 16 or 32 links, W lanes each, one link per lane: equal
// modules meet in the group's slots of the warp's table, and the lane that
// filled a slot evaluates its module. base: the warp's first record. Loads are
// issued for every lane (those past the unit's links read its first), so that
// none waits on a branch.
__device__ __forceinline__ void eval_small(const StageDev &a, const SubCtx &sc, int W, int base, int end, int tab) {
    const int lane = threadIdx.x & 31, gl = lane & (W - 1);
    const int i = base + lane / W;
    const bool valid = i < end;
    const URec r = load_rec(a.urec + (valid ? i : base));
    const int d = r.dout + r.din;
    const bool has = valid && gl < d;
    int32_t nbr = 0, key = -1;
    fx_t v = 0;
    if (d > 0) {
        const int j = has ? gl : 0;
        bool isout;
        const uint32_t e = link_at(r, j, isout);
        nbr = (isout ? a.out_dst : a.in_src)[e];
        v = (isout ? a.out_fx : a.in_fx)[e];
        key = a.mod[nbr];
    }
    const Stat4 ua = load_stat(a.attr + r.u);
    const ModRec mA = load_mod(a.rec + r.A);
    const double DA = a.rec[r.A].D;
    const int32_t nA = a.mcount[r.A];
    const double se = unit_sum_exit(a, sc, r.u);
    const bool other = has && key != r.A;
    const int tb = tab + (lane / W) * 4 * W, mask = 4 * W - 1;
    int slot = tb;
    bool fresh = false;
    ModRec rm = mA;
    if (other) {
        rm = load_mod(a.rec + key);
        int s = tab_slot(key, mask);
        int32_t prev = atomicCAS(&slot_key(tb + s), kEmpty, key);
        for (int probe = 0; prev != kEmpty && prev != key && probe < mask; probe++) {  // at most a quarter full
            s = (s + 1) & mask;
            prev = atomicCAS(&slot_key(tb + s), kEmpty, key);
        }
        slot = tb + s;
        fresh = prev == kEmpty;
        add_slot(slot, v);
    }
    fx_t sA = has && !other ? v : 0;
    for (int o = W / 2; o > 0; o >>= 1) sA += __shfl_xor_sync(kFull, sA, o);
    __syncwarp();
    double new_exit, new_stay;
    const UnitCtx c = make_ctx_lanes(W, ua, mA, DA, se, r.A, sA, gl, new_exit, new_stay);
    double best = 0.0;
    int32_t bm = INT_MAX;
    if (fresh) {
        best = candidate_delta(c, rm, take_slot(slot), plogp2);
        bm = key;
    }
    // a lane without a candidate holds (0, INT_MAX), which no candidate that can win loses to
    for (int o = W / 2; o > 0; o >>= 1) {
        const double ob2 = __shfl_xor_sync(kFull, best, o);
        const int32_t om = __shfl_xor_sync(kFull, bm, o);
        if (better(ob2, om, best, bm)) {
            best = ob2;
            bm = om;
        }
    }
    if (valid && decide(a, sc, i, r.u, c, nA, new_exit, new_stay, best, bm, gl == 0) && a.prior && has)
        a.next_active[nbr] = 1;
    __syncwarp();
}

struct TeamShared {
    fx_t sA[kSwWarps];
    double best[kSwWarps];
    int32_t mod[kSwWarps];
    fx_t dA[kSwWarps], dT[kSwWarps];
    unsigned next[kSwWarps];
};

// One unit evaluated by a team of NW = 1, 4 or 16 warps through the team's slice
// of the block's table (from slot tab on). The table is empty before and after every unit: each
// warp empties the slots it filled while it evaluates them.
__device__ __forceinline__ void eval_team(const StageDev &a, const SubCtx &sc, int NW, int i, int tab, TeamShared &sh) {
    const int w = threadIdx.x >> 5, w0 = w & ~(NW - 1), lane = threadIdx.x & 31, rank = threadIdx.x - w0 * 32;
    const int NT = NW * 32, bar = team_bar(NW, w0);
    const URec r = load_rec(a.urec + i);
    const int d = r.dout + r.din;
    const int mask = NW * kWarpTab - 1;  // the team's whole slice: at least two slots per link
    const Stat4 ua = load_stat(a.attr + r.u);
    const int32_t nA = a.mcount[r.A];
    const double se = unit_sum_exit(a, sc, r.u);
    // links j = rank, rank + NT, ...: those to the unit's own module are summed, the others go to
    // the table; slots that this warp fills go to its list
    fx_t sA = 0;
    int cnt = 0;
    for (int j0 = 0; j0 < d; j0 += kIlp * NT) {
        int32_t key[kIlp];
        fx_t q[kIlp];
#pragma unroll
        for (int k = 0; k < kIlp; k++) {
            key[k] = -1;
            q[k] = 0;
            if (j0 + k * NT < d) {  // the same in the whole team
                const int j = min(j0 + k * NT + rank, d - 1);
                bool isout;
                const uint32_t e = link_at(r, j, isout);
                key[k] = (isout ? a.out_dst : a.in_src)[e];
                q[k] = (isout ? a.out_fx : a.in_fx)[e];
            }
        }
#pragma unroll
        for (int k = 0; k < kIlp; k++)
            if (j0 + k * NT < d) key[k] = a.mod[key[k]];
        int slot[kIlp];
        int32_t prev[kIlp];
#pragma unroll
        for (int k = 0; k < kIlp; k++) {
            if (j0 + k * NT + rank >= d) key[k] = -1;
            if (key[k] == r.A) {
                sA += q[k];
                key[k] = -1;
            }
            slot[k] = tab + tab_slot(key[k], mask);
            prev[k] = 0;
            if (key[k] >= 0) prev[k] = atomicCAS(&slot_key(slot[k]), kEmpty, key[k]);
        }
        // at least twice as many slots as links: a free one exists
        for (int probe = 0; probe < mask; probe++) {
            bool more = false;
#pragma unroll
            for (int k = 0; k < kIlp; k++)
                if (key[k] >= 0 && prev[k] != kEmpty && prev[k] != key[k]) {
                    slot[k] = tab + ((slot[k] - tab + 1) & mask);
                    prev[k] = atomicCAS(&slot_key(slot[k]), kEmpty, key[k]);
                    more = true;
                }
            if (!more) break;
        }
        unsigned old[kIlp];
        int nf = 0;
#pragma unroll
        for (int k = 0; k < kIlp; k++) {
            old[k] = 0;
            if (key[k] >= 0) old[k] = atomicAdd(&slot_lo(slot[k]), (unsigned)q[k]);
            if (prev[k] != kEmpty) prev[k] = 0;  // prev: kEmpty for a slot this lane filled
            nf -= prev[k];
        }
#pragma unroll
        for (int k = 0; k < kIlp; k++)
            if (key[k] >= 0)
                atomicAdd(&slot_hi(slot[k]), (unsigned)((unsigned long long)q[k] >> 32) +
                                              (old[k] + (unsigned)q[k] < old[k] ? 1u : 0u));
        int x = nf;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, x, o);
            if (lane >= o) x += y;
        }
        int pos = cnt + x - nf;
#pragma unroll
        for (int k = 0; k < kIlp; k++)
            if (prev[k] == kEmpty) warp_list(pos++) = (uint16_t)slot[k];
        cnt += __shfl_sync(kFull, x, 31);
    }
    const ModRec mA = load_mod(a.rec + r.A);
    const double DA = a.rec[r.A].D;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sA += __shfl_xor_sync(kFull, sA, o);
    if (lane == 0) sh.sA[w] = sA;
    team_sync(NW, bar);
    if (NW > 1) {
        sA = 0;
        for (int q = 0; q < NW; q++) sA += sh.sA[w0 + q];
    }
    double new_exit, new_stay;
    const UnitCtx c = make_ctx_lanes(32, ua, mA, DA, se, r.A, sA, lane, new_exit, new_stay);
    double best = 0.0;
    int32_t bm = INT_MAX;
    for (int q = lane; q < cnt; q += 32) {
        const int s = warp_list(q);
        const int32_t m = slot_key(s);
        const ModRec rm = load_mod(a.rec + m);
        const double dl = candidate_delta(c, rm, take_slot(s), plogp2);
        if (better(dl, m, best, bm)) {
            best = dl;
            bm = m;
        }
    }
    warp_best(best, bm);
    if (lane == 0) {
        sh.best[w] = best;
        sh.mod[w] = bm;
    }
    team_sync(NW, bar);
    if (NW > 1) {
        best = lane < NW ? sh.best[w0 + lane] : 0.0;
        bm = lane < NW ? sh.mod[w0 + lane] : INT_MAX;
        warp_best(best, bm);
    }
    if (decide(a, sc, i, r.u, c, nA, new_exit, new_stay, best, bm, rank == 0) && a.prior) {
        for (int j = rank; j < d; j += NT)
            a.next_active[j < r.dout ? a.out_dst[r.ob + j] : a.in_src[r.ib + (j - r.dout)]] = 1;
    }
}

// The module unit u moves to: p its proposal; -1 if it stays (a lost bid).
__device__ __forceinline__ int32_t resolve(const StageDev &a, uint32_t stamp, int32_t u, int32_t p) {
    if (p >= 0 || p == -1) return p;
    const int32_t m = -(p + 3);
    return __ldcg(a.claim + m) == claim_key(stamp, u) ? m : -1;
}

// Changes of OUT[A] and OUT[T] from the links of mover u (delta_links of
// rmx_moves.cu, with memberships not yet updated: a neighbour's new module
// comes from its proposal).
__device__ __forceinline__ void move_links(const StageDev &a, int NT, uint32_t stamp, const URec &r, int32_t T, int rank,
                                           fx_t &dA, fx_t &dT) {
    const int d = r.dout + r.din;
    for (int j0 = rank; j0 < d; j0 += kIlp * NT) {
        int32_t w[kIlp], b[kIlp];
        fx_t q[kIlp];
        uint32_t st[kIlp];
#pragma unroll
        for (int k = 0; k < kIlp; k++) {
            const int j = j0 + k * NT;
            w[k] = -1;
            if (j < d) {
                bool isout;
                const uint32_t e = link_at(r, j, isout);
                w[k] = isout ? a.out_dst[e] : a.in_src[e];
                q[k] = isout ? a.out_fx[e] : a.in_fx[e];
            }
        }
#pragma unroll
        for (int k = 0; k < kIlp; k++)
            if (w[k] >= 0) {
                b[k] = a.mod[w[k]];
                st[k] = a.stamp[w[k]];
            }
#pragma unroll
        for (int k = 0; k < kIlp; k++) {
            if (w[k] < 0) continue;
            const int32_t nw = st[k] == stamp ? resolve(a, stamp, w[k], a.prop[w[k]]) : -1;
            if (j0 + k * NT < r.dout) {
                if (r.A != b[k]) dA -= q[k];
                if (T != (nw >= 0 ? nw : b[k])) dT += q[k];
            } else if (nw < 0) {  // a moving source counts the link itself
                if (b[k] == r.A)
                    dA += q[k];
                else if (b[k] == T)
                    dT -= q[k];
            }
        }
    }
}

// The statistics of A and T change by mover u: eight lanes, one atomic each.
__device__ __forceinline__ void move_stats(const StageDev &a, const URec &r, int32_t T, bool bid, int l8, fx_t dA,
                                           fx_t dT) {
    const bool to = l8 < 4;
    const int f = l8 & 3;
    fx_t v = f == 3 ? 0 : reinterpret_cast<const fx_t *>(a.attr + r.u)[f];
    v = f == 3 ? (to ? dT : dA) : (to ? v : -v);
    if (v) atomic_add_fx(reinterpret_cast<fx_t *>(a.stat + (to ? T : r.A)) + f, v);
    if (l8 == 0) {
        atomicAdd(a.mcount + T, 1);
        if (bid) a.minst[T] = a.uinst[r.u];
    }
    if (l8 == 4) atomicSub(a.mcount + r.A, 1);
}

// Movers among records beg..end of at most 128 links, W = 8 or 32 lanes each.
// Warps take runs of records, as short as spreads them over all warps.
__device__ __forceinline__ void apply_light(const StageDev &a, uint32_t stamp, int W, int beg, int end, int wid, int nw) {
    if (beg >= end) return;
    const int lane = threadIdx.x & 31, g = lane / W, gl = lane & (W - 1), G = 32 / W;
    int per = (end - beg + nw - 1) / nw;
    per = per > 32 ? 32 : (per < G ? G : per);
    for (int64_t b0 = beg + (int64_t)wid * per; b0 < end; b0 += (int64_t)nw * per) {
        const int i = (int)b0 + lane;
        int32_t p = -1, T = -1;
        if (lane < per && i < end) {
            p = a.tgt[i];
            T = p < -1 ? resolve(a, stamp, a.urec[i].u, p) : p;
        }
        for (unsigned mk = __ballot_sync(kFull, T >= 0); mk;) {
            unsigned m = mk;
            for (int q = 0; q < G; q++) {
                if (q < g) m &= m - 1;
                mk &= mk - 1;
            }
            const int src = m ? __ffs(m) - 1 : 0;
            const int32_t t = __shfl_sync(kFull, T, src), pp = __shfl_sync(kFull, p, src);
            fx_t dA = 0, dT = 0;
            URec r = {};
            if (m) {
                r = load_rec(a.urec + b0 + src);
                move_links(a, W, stamp, r, t, gl, dA, dT);
            }
            for (int o = W / 2; o > 0; o >>= 1) {
                dA += __shfl_xor_sync(kFull, dA, o);
                dT += __shfl_xor_sync(kFull, dT, o);
            }
            if (m && gl < 8) move_stats(a, r, t, pp < -1, gl, dA, dT);
        }
    }
}

// Heavier movers, a team of NW = 4 or 16 warps each.
__device__ __forceinline__ void apply_team(const StageDev &a, uint32_t stamp, int NW, int beg, int end, int id,
                                           int teams, TeamShared &sh) {
    const int w = threadIdx.x >> 5, w0 = w & ~(NW - 1), lane = threadIdx.x & 31, rank = threadIdx.x - w0 * 32;
    const int bar = team_bar(NW, w0);
    for (int i = beg + id; i < end; i += teams) {
        const int32_t p = a.tgt[i];
        if (p == -1) continue;
        const URec r = load_rec(a.urec + i);
        const int32_t T = resolve(a, stamp, r.u, p);
        if (T < 0) continue;
        fx_t dA = 0, dT = 0;
        move_links(a, NW * 32, stamp, r, T, rank, dA, dT);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            dA += __shfl_xor_sync(kFull, dA, o);
            dT += __shfl_xor_sync(kFull, dT, o);
        }
        if (lane == 0) {
            sh.dA[w] = dA;
            sh.dT[w] = dT;
        }
        team_sync(NW, bar);
        if (rank < 8) {
            dA = dT = 0;
            for (int q = 0; q < NW; q++) {
                dA += sh.dA[w0 + q];
                dT += sh.dT[w0 + q];
            }
            move_stats(a, r, T, p < -1, rank, dA, dT);
        }
        team_sync(NW, bar);  // the sums are read before the next unit's are written
    }
}

// The evaluation of one sub-batch. bo: its bins' bounds among the records;
// next: its bins' work counters. If every unit can have warps of its own at
// once, units are dealt out (wide: 4 warps for a warp-bin unit and 16 for a
// mid or block unit, where that fits too); otherwise teams take the next unit
// of the heaviest bin that has one left. Every unit goes through one of the two
// evaluations below, each compiled once: the kernel's code stays small enough
// for the instruction caches, which a sub-batch of few units runs through only
// once.
__device__ __forceinline__ void eval_subbatch(const StageDev &a, const SubCtx &sc, const unsigned *bo, unsigned *next,
                                              TeamShared &sh) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nb = (int)gridDim.x, bx = (int)blockIdx.x;
    const int n1 = (int)(bo[kBinMid] - bo[kBinWarp]), n32 = (int)(bo[kBinWarp] - bo[kBinReg32]),
              w16 = (int)(bo[kBinReg32] - bo[kBinReg16] + 1) / 2, w8 = (int)(bo[kBinReg16] - bo[kBinReg8] + 3) / 4,
              n4 = (int)(bo[kBinLarge] - bo[kBinMid]), nl = (int)(bo[kBinHub] - bo[kBinLarge]);
    const int small = w8 + w16 + n32, light = n1 + small;
    const int rw = nb - nl - n4, rn = nb - nl;  // blocks left by the 16-warp units: wide, narrow
    const bool wide = rw >= 0 && n1 <= 4 * rw && 4 * n1 + small <= 16 * rw;
    const bool fits = wide || (rn >= 0 && n4 <= 4 * rn && 4 * n4 + light <= 16 * rn);
    int phase = fits ? 3 : nl > 0 ? 0 : n4 > 0 ? 1 : 2;
    int x = 0;  // the warp's place among the light bins' work
    bool first = true;
    for (;;) {
        int NW = 0;        // warps of the unit's team; 0: the light bins' work x
        int i = 0;         // its record
        if (phase == 3) {
            const int u16 = wide ? nl + n4 : nl, u4 = wide ? n1 : n4, R = nb - u16;
            const int q = (w >> 2) * R + (bx - u16);  // this warp's 4-warp slot
            if (bx < u16) {
                NW = 16;
                i = (int)bo[kBinHub] - 1 - bx;
            } else if (q < u4) {
                NW = 4;
                i = (int)bo[wide ? kBinWarp : kBinMid] + q;
            } else {
                x = (wide ? n1 : 0) + (w & 3) * (4 * R - u4) + (q - u4);
            }
        } else if (phase == 0) {
            __syncthreads();
            if (threadIdx.x == 0) sh.next[0] = atomicAdd(next + 2, 1u);
            __syncthreads();
            const unsigned k = sh.next[0];
            if (k >= (unsigned)nl) {
                phase = n4 > 0 ? 1 : 2;
                __syncthreads();
                continue;
            }
            NW = 16;
            i = (int)bo[kBinLarge] + k;
        } else if (phase == 1) {
            const int bar = team_bar(4, w & ~3);
            if ((threadIdx.x & 127) == 0) sh.next[w] = atomicAdd(next + 1, 1u);
            team_sync(4, bar);
            const unsigned k = sh.next[w & ~3];
            team_sync(4, bar);
            if (k >= (unsigned)n4) {
                phase = 2;
                continue;
            }
            NW = 4;
            i = (int)bo[kBinLarge] - 1 - k;
        } else {
            unsigned y = 0;
            if (first) {
                if (lane == 0) y = atomicAdd(next, 1u);
                x = (int)__shfl_sync(kFull, y, 0);
                first = false;
            }
        }
        unsigned ahead = 0;  // the next work of a light phase is taken before this one is done
        if (phase == 2) {
            if (x >= light) break;
            if (lane == 0) ahead = atomicAdd(next, 1u);
        }
        int W = 0;
        if (NW == 0) {
            int y = x;
            if (y < n1) {
                NW = 1;
                i = (int)bo[kBinWarp] + y;
            } else if ((y -= n1) < n32) {
                W = 32;
                i = (int)bo[kBinReg32] + y;
            } else if ((y -= n32) < w16) {
                W = 16;
                i = (int)bo[kBinReg16] + 2 * y;
            } else if ((y -= w16) < w8) {
                W = 8;
                i = (int)bo[kBinReg8] + 4 * y;
            }
        }
        if (NW > 0)
            eval_team(a, sc, NW, i, (w & ~(NW - 1)) * kWarpTab, sh);
        else if (W > 0)
            eval_small(a, sc, W, i, bo[W == 32 ? kBinWarp : W == 16 ? kBinReg32 : kBinReg16], w * kWarpTab);
        if (phase == 3) break;
        if (phase == 2) x = (int)__shfl_sync(kFull, ahead, 0);
    }
}

__device__ __forceinline__ int bin_of(const BinBounds &bb, int64_t d) {
    return d <= 8           ? kBinReg8
           : d <= 16        ? kBinReg16
           : d <= 32        ? kBinReg32
           : d <= bb.warp   ? kBinWarp
           : d <= bb.mid    ? kBinMid
           : d <= bb.block  ? kBinBlock
           : d <= bb.large  ? kBinLarge
                            : kBinHub;
}

// Sum over the block, returned to every thread (ws: 32 words).
__device__ __forceinline__ fx_t block_sum_all(fx_t v, fx_t *ws) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
    __syncthreads();
    fx_t t = 0;
#pragma unroll
    for (int q = 0; q < kSwWarps; q++) t += ws[q];
    return t;
}

__global__ void __launch_bounds__(kSwT, RMX_STAGE_MINB) k_stage(const __grid_constant__ StageDev a) {
    cg::grid_group grid = cg::this_grid();
    __shared__ TeamShared sh;
    __shared__ unsigned hist[kMaxBuckets], base[kMaxBuckets];
    __shared__ unsigned boff[kMaxBuckets + 1];
    __shared__ fx_t ws[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nb = (int)gridDim.x, bx = (int)blockIdx.x;
    const int64_t gtid = (int64_t)bx * kSwT + threadIdx.x, gthreads = (int64_t)nb * kSwT;
    const int nbk = a.nsub * kBins;
    for (int s = threadIdx.x; s < kSwTab; s += kSwT) {
        slot_key(s) = kEmpty;
        slot_lo(s) = 0;
        slot_hi(s) = 0;
    }
    // the block's run of module ids in the list of empty modules
    const int64_t fchunk = (((int64_t)a.cap + nb - 1) / nb + kSwT - 1) / kSwT * kSwT;
    const int64_t f0 = min((int64_t)a.cap, (int64_t)bx * fchunk), f1 = min((int64_t)a.cap, f0 + fchunk);
    double Lcur = a.K == 1 ? a.L[0] : 0.0, se1 = a.K == 1 ? a.sum_exit[0] : 0.0;
    int iter = 0;
    for (;;) {
        SweepSet *const set = a.set + (iter & 1);
        const uint32_t seed = mix_seed(a.run_seed, a.sweep0 + (uint64_t)iter + 1);
        const bool all = iter == 0 || !a.prior;
        // ---- count
        for (int k = threadIdx.x; k < nbk; k += kSwT) hist[k] = 0;
        __syncthreads();
        for (int64_t u = gtid; u < a.n; u += gthreads) {
            if (!all && !a.next_active[u]) continue;
            if (a.K > 1 && !a.active[a.uinst[u]]) continue;
            const int64_t d = (a.out_off[u + 1] - a.out_off[u]) + (a.in_off[u + 1] - a.in_off[u]);
            const int sb = a.nsub > 1 ? (int)(mix32((uint32_t)u ^ seed) % (uint32_t)a.nsub) : 0;
            atomicAdd(hist + sb * kBins + bin_of(a.bb, d), 1u);
        }
        if (a.allow_new) {
            fx_t c = 0;
            for (int64_t m = f0 + threadIdx.x; m < f1; m += kSwT) c += a.mcount[m] == 0;
            c = block_sum_all(c, ws);
            if (threadIdx.x == 0) a.free_cnt[bx] = (int32_t)c;
        }
        __syncthreads();
        for (int k = threadIdx.x; k < nbk; k += kSwT)
            if (hist[k]) atomicAdd(set->cnt + k, hist[k]);
        grid.sync();
        // ---- fill
        if (w == 0) {  // bucket offsets
            unsigned run = 0;
            for (int k0 = 0; k0 < nbk; k0 += 32) {
                const unsigned c = k0 + lane < nbk ? __ldcg(set->cnt + k0 + lane) : 0u;
                unsigned x = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned y = __shfl_up_sync(kFull, x, o);
                    if (lane >= o) x += y;
                }
                if (k0 + lane < nbk) boff[k0 + lane] = run + x - c;
                run += __shfl_sync(kFull, x, 31);
            }
            if (lane == 0) boff[nbk] = run;
        }
        for (int k = threadIdx.x; k < nbk; k += kSwT)
            if (hist[k]) base[k] = atomicAdd(set->cur + k, hist[k]);
        int64_t n_free = 0;
        if (a.allow_new) {
            fx_t before = 0, tot = 0;
            for (int64_t b = threadIdx.x; b < nb; b += kSwT) {
                const fx_t c = __ldcg(a.free_cnt + b);
                tot += c;
                if (b < bx) before += c;
            }
            n_free = block_sum_all(tot, ws);
            int64_t pos = block_sum_all(before, ws);
            for (int64_t m0 = f0; m0 < f1; m0 += kSwT) {  // ascending within the block's run
                const int64_t m = m0 + threadIdx.x;
                const bool e = m < f1 && a.mcount[m] == 0;
                const unsigned bal = __ballot_sync(kFull, e);
                __syncthreads();
                if (lane == 0) ws[w] = __popc(bal);
                __syncthreads();
                int64_t q = pos + __popc(bal & ((1u << lane) - 1u));
                fx_t sum = 0;
#pragma unroll
                for (int k = 0; k < kSwWarps; k++) {
                    if (k < w) q += ws[k];
                    sum += ws[k];
                }
                if (e) a.free_list[q] = (int32_t)m;
                pos += sum;
            }
        }
        __syncthreads();
        for (int64_t u = gtid; u < a.n; u += gthreads) {
            if (a.prior) {
                const bool was = all || a.next_active[u];
                a.next_active[u] = 0;
                if (!was) continue;
            }
            if (a.K > 1 && !a.active[a.uinst[u]]) continue;
            URec r = {};
            const int64_t ob = a.out_off[u], ib = a.in_off[u];
            const int64_t dout = a.out_off[u + 1] - ob, din = a.in_off[u + 1] - ib;
            r.ob = (uint32_t)ob;
            r.ib = (uint32_t)ib;
            const int sb = a.nsub > 1 ? (int)(mix32((uint32_t)u ^ seed) % (uint32_t)a.nsub) : 0;
            const int k = sb * kBins + bin_of(a.bb, dout + din);
            r.u = (int32_t)u;
            r.A = a.mod[u];
            r.dout = (int32_t)dout;
            r.din = (int32_t)din;
            a.urec[boff[k] + atomicAdd(base + k, 1u)] = r;
        }
        {  // the other set, last read before this sweep's first barrier, is cleared for the next sweep
            SweepSet *const other = a.set + 1 - (iter & 1);
            if (bx == 0) {
                for (int k = threadIdx.x; k < nbk; k += kSwT) other->cnt[k] = other->cur[k] = 0;
                if (threadIdx.x < kMaxSub)
                    other->any[threadIdx.x] = other->next[threadIdx.x][0] = other->next[threadIdx.x][1] =
                        other->next[threadIdx.x][2] = 0;
                if (threadIdx.x < 3) other->acc[threadIdx.x] = 0;
                if (threadIdx.x == 0) other->remaining = 0;
            }
            if (a.K > 1)
                for (int64_t k = gtid; k < 3 * (int64_t)a.K; k += gthreads) a.acc[k] = 0;
        }
        grid.sync();
        // ---- sub-batches
        for (int sb = 0; sb < a.nsub; sb++) {
            const unsigned *const bo = boff + sb * kBins;
            SubCtx sc;
            sc.stamp = a.stamp0 + (uint32_t)(iter * a.nsub + sb + 1);
            sc.hseed = mix_seed(seed, (uint64_t)sb);
            sc.n_free = n_free;
            sc.any = set->any + sb;
            sc.sum_exit = se1;
            eval_subbatch(a, sc, bo, set->next[sb], sh);
            grid.sync();
            if (!__ldcg(set->any + sb)) continue;  // the same in every block: nothing moves
            for (int h = 0; h < 2; h++) {
                apply_team(a, sc.stamp, h ? 4 : 16, bo[h ? kBinMid : kBinLarge], bo[h ? kBinLarge : kBinHub],
                           h ? (w / 4) * nb + bx : bx, h ? 4 * nb : nb, sh);
                __syncthreads();
            }
            for (int h = 0; h < 2; h++)
                apply_light(a, sc.stamp, h ? 8 : 32, bo[h ? kBinReg8 : kBinWarp], bo[h ? kBinWarp : kBinMid],
                            w * nb + bx, nb * kSwWarps);
            grid.sync();
            // the hub bin, which the evaluation has no part for and so proposes nothing, is left out (the host
            // takes no level with hub units here)
            for (int64_t i = bo[0] + gtid; i < bo[kBinHub]; i += gthreads) {
                const int32_t p = a.tgt[i];
                if (p == -1) continue;
                const int32_t u = a.urec[i].u, A = a.urec[i].A;
                const int32_t T = resolve(a, sc.stamp, u, p);
                if (T < 0) continue;
                a.mod[u] = T;
                write_terms(a.stat, a.term, a.rec, A);
                write_terms(a.stat, a.term, a.rec, T);
            }
            grid.sync();
        }
        // ---- code length and stop rule
        fx_t t0 = 0, t1 = 0, t2 = 0;
        for (int64_t m = gtid; m < a.cap; m += gthreads) {
            if (a.mcount[m] <= 0) continue;
            const Stat4 st = load_stat(a.stat + m);
            const double P = from_fx(st.P);
            const double e = exit_flow(P, from_fx(st.TW), from_fx(st.D), from_fx(st.OUT));
            const double2 tm = a.term[m];
            const fx_t a0 = to_fxl(e), a1 = to_fxl(tm.x), a2 = to_fxl(tm.y);
            if (a.K == 1) {
                t0 += a0;
                t1 += a1;
                t2 += a2;
            } else {
                fx_t *const p = a.acc + 3 * (int64_t)a.minst[m];
                atomic_add_fx(p, a0);
                atomic_add_fx(p + 1, a1);
                atomic_add_fx(p + 2, a2);
            }
        }
        bool go;
        if (a.K == 1) {
            t0 = block_sum_all(t0, ws);
            t1 = block_sum_all(t1, ws);
            t2 = block_sum_all(t2, ws);
            if (threadIdx.x < 3) {
                const fx_t v = threadIdx.x == 0 ? t0 : threadIdx.x == 1 ? t1 : t2;
                if (v) atomic_add_fx(set->acc + threadIdx.x, v);
            }
            grid.sync();
            se1 = from_fxl(__ldcg(set->acc));
            const double L = plogp(se1) - 2.0 * from_fxl(__ldcg(set->acc + 1)) + from_fxl(__ldcg(set->acc + 2)) -
                             from_fxl(a.s0[0]);
            const double dl = Lcur - L;
            go = a.subtune ? !(dl / a.ln2 < a.threshold) : !(dl >= 0 && dl / a.ln2 < a.threshold);
            Lcur = L;
        } else {
            grid.sync();
            unsigned long long c = 0;
            for (int64_t k = gtid; k < a.K; k += gthreads) {
                const double se = from_fxl(__ldcg(a.acc + 3 * k));
                const double L = plogp(se) - 2.0 * from_fxl(__ldcg(a.acc + 3 * k + 1)) +
                                 from_fxl(__ldcg(a.acc + 3 * k + 2)) - from_fxl(a.s0[k]);
                const double old = a.L[k];
                a.sum_exit[k] = se;
                a.L[k] = L;
                if (!a.active[k]) continue;
                const double dl = old - L;
                const bool stop = a.subtune ? dl / a.ln2 < a.threshold : (dl >= 0 && dl / a.ln2 < a.threshold);
                if (stop)
                    a.active[k] = 0;
                else
                    c++;
            }
            c = (unsigned long long)block_sum_all((fx_t)c, ws);
            if (threadIdx.x == 0 && c) atomicAdd(&set->remaining, c);
            grid.sync();
            go = __ldcg(&set->remaining) > 0;
        }
        iter++;
        if (!go || iter >= a.max_iter) break;  // the same in every block
    }
    if (gtid == 0) {
        a.ctl[0] = iter;
        if (a.K == 1) {
            a.sum_exit[0] = se1;
            a.L[0] = Lcur;
        }
    }
}

}  // namespace

size_t fused_stage_bytes(int32_t n) {
    return (size_t)n * (sizeof(URec) + sizeof(int32_t)) + 2 * sizeof(SweepSet) + (1 << 16);
}

void fused_stage(const Level &lv, ModState &M, InstState &I, SweepWork &W, const FusedStage &f, int64_t *ctl, Arena &ar,
                 cudaStream_t s) {
    static std::mutex mu;
    static std::vector<int> resident;  // per device: resident blocks per SM
    int dev = 0, per_sm = 0;
    RMX_CUDA(cudaGetDevice(&dev));
    {
        std::lock_guard<std::mutex> lk(mu);
        if ((int)resident.size() <= dev) resident.resize(dev + 1, 0);
        if (resident[dev] == 0) {
            RMX_CUDA(cudaFuncSetAttribute(k_stage, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStageSmem));
            RMX_CUDA(cudaFuncSetAttribute(k_stage, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
            RMX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident[dev], k_stage, kSwT, kStageSmem));
        }
        per_sm = resident[dev];
    }
    if (per_sm < 1) throw CudaError(cudaErrorLaunchOutOfResources, "stage kernel does not fit an SM");
    const size_t mk = ar.mark();
    StageDev a;
    a.n = lv.n;
    a.out_off = lv.out_off;
    a.in_off = lv.in_off;
    a.out_dst = lv.out_dst;
    a.in_src = lv.in_src;
    a.out_fx = lv.out_fx;
    a.in_fx = lv.in_fx;
    a.attr = lv.attr;
    a.mod = lv.mod;
    a.uinst = lv.inst;
    a.cap = M.cap;
    a.stat = M.stat;
    a.term = M.term;
    a.rec = M.rec;
    a.mcount = M.count;
    a.minst = M.inst;
    a.K = I.n;
    a.sum_exit = I.sum_exit;
    a.L = I.L;
    a.s0 = I.s0;
    a.acc = I.acc;
    a.active = I.active;
    a.urec = ar.alloc<URec>(lv.n);
    a.tgt = ar.alloc<int32_t>(lv.n);
    a.prop = W.prop;
    a.stamp = W.stamp;
    a.next_active = W.next_active;
    a.free_list = W.free_list;
    a.claim = W.claim;
    a.prior = f.prior;
    a.allow_new = f.allow_new;
    a.subtune = f.subtune;
    a.max_iter = f.max_iter;
    a.nsub = f.nsub;
    a.vthresh = f.vthresh;
    a.threshold = f.threshold;
    a.ln2 = f.ln2;
    a.run_seed = f.run_seed;
    a.stamp0 = f.stamp;
    a.sweep0 = f.sweep_no;
    a.bb = BinBounds{W.tune.warp_max, W.tune.mid_max, W.tune.block_max, W.tune.large_max};
    a.set = ar.alloc<SweepSet>(2);
    a.ctl = ctl;
    // Enough blocks that every warp of a sub-batch's evaluation has about four units or 128
    // links; fewer make the grid barriers cheaper.
    const int64_t full = (int64_t)std::min(per_sm, 2) * num_sms();
    const int64_t want = std::max<int64_t>({(int64_t)lv.n / 16, lv.m / 2048, (int64_t)M.cap / 4096, 1});
    const int nb = (int)std::min(full, want);
    a.free_cnt = ar.alloc<int32_t>(nb);
    RMX_CUDA(cudaMemsetAsync(a.set, 0, sizeof(SweepSet) * 2, s));
    void *args[] = {(void *)&a};
    RMX_CUDA(cudaLaunchCooperativeKernel((void *)k_stage, dim3(nb), dim3(kSwT), args, kStageSmem, s));
    RMX_LAUNCHED();
    ar.release(mk);
}

}  // namespace rmx

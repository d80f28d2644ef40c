// Conversion of a partition into the next super-node level as one cooperative
// launch: convertModulesToSuperNodes (Module.cpp:3008-3077) and
// generateSuperNodesFromSubModules (Module.cpp:3083-3158), for levels of up to
// a few million links.
//
// The multi-kernel path (convert_to_supernodes in rmx_engine.cu,
// aggregate_links in rmx_coarsen.cu) takes about 35 launches and five host
// round trips, 0.2 ms on any level however small. Here one persistent grid goes
// through the same steps with a grid barrier after each:
//   units per module; modules numbered in ascending order (the super-nodes,
//   with the module's statistics); each row's group; room for each group's
//   links; links between groups gathered there; each group's links summed by
//   destination in a shared-memory table; CSR and CSC offsets; CSR rows and,
//   column by column, CSC entries.
// Bound by the barriers (11 of 1.25 us) and each step's chain of dependent
// accesses: 0.22 -> 0.075 ms on the 1000-node planted graph. On levels of
// millions of links by the atomics: of 0.5 ms for 7.6M links, gathering takes
// 0.11, the sums 0.13 to 0.2 and the rows and columns 0.1 (0.3 and 0.3 where the
// groups are 290,000 sub-modules).
// Link sums are exact integers, rows and columns come in no particular order.
// A group whose links do not fit the tables is left to the other path: the
// kernel reports it and nothing it wrote is kept.
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "rmx_moves.cuh"

namespace cg = cooperative_groups;

namespace rmx {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kCvT = 512, kCvWarps = kCvT / 32, kCvTab = 8192, kCvWarpTab = kCvTab / kCvWarps;
constexpr int kCvList = 256;             // slots a warp can have filled
constexpr int kCvIlp = 4;
// Blocks per SM. With one, larger levels wait on the sums' shared-memory and
// column atomics: all conversions of a run on 250,001 nodes 15.3 ms, with two
// (64 registers, 68 bytes a thread spilt) 14.9; on 400,001 nodes 39.1 and 37.9.
constexpr int kCvBlocks = 2;
// links of a group summed by a warp, four warps, a block in one pass, a block in several
constexpr int kCvWarpMax = 256, kCvTeamMax = 1024, kCvBlockMax = 4096, kCvMost = 16384;
constexpr size_t kCvSmem = (size_t)kCvTab * 12 + (size_t)kCvWarps * kCvList * sizeof(uint16_t);

struct ConvDev {
    int32_t N;
    const int32_t *unit_mod;      // module of every node
    int32_t *count;               // nodes per module (written here)
    const Stat4 *stat;
    const int32_t *minst, *parent_inst;
    int sub, K;
    // source level
    int32_t n;
    int64_t m;
    const int64_t *off;
    const int32_t *dst, *src;
    const fx_t *fx;
    const int32_t *row_mod;       // module of every source unit (null: the source units are the nodes)
    // new level
    int32_t *mod, *nnodes, *inst, *node_sn;
    Stat4 *attr;
    int64_t *out_off, *in_off;
    int32_t *out_dst, *out_src, *in_src;
    fx_t *out_fx, *in_fx;
    // scratch
    int32_t *snid, *group;
    unsigned *gcap, *gloff, *gcross, *rowlen, *colcnt;
    int32_t *sk, *rk;             // gathered links and summed rows: destination group (sk then: place in its column)
    fx_t *sq, *rq;                //   and flow
    int32_t *list;                // 3 x N: groups by the size of their team
    int64_t *blk;                 // 2 per block
    // [0] super-nodes [1] links [2] a group has too many links [3..6] hub units, partitions, links, chunks
    // [8..10] groups per list [11] gathered links allotted [12] groups of the block list taken
    // [13] a list of filled slots overflowed. A word that the blocks test after a barrier is not written again before
    // the next one: a block still on its way to the test would leave alone, and the others wait for it.
    unsigned long long *ctl;
    int64_t hub_bound, hub_part, hub_chunk, hub_max_parts;
};

extern __shared__ __align__(16) unsigned char conv_smem[];
__device__ __forceinline__ int32_t &cv_key(int s) { return reinterpret_cast<int32_t *>(conv_smem)[s]; }
__device__ __forceinline__ unsigned &cv_lo(int s) { return reinterpret_cast<unsigned *>(conv_smem)[kCvTab + s]; }
__device__ __forceinline__ unsigned &cv_hi(int s) { return reinterpret_cast<unsigned *>(conv_smem)[2 * kCvTab + s]; }
__device__ __forceinline__ uint16_t &cv_list(int k) {
    return reinterpret_cast<uint16_t *>(conv_smem + (size_t)kCvTab * 12)[(threadIdx.x >> 5) * kCvList + k];
}

struct ConvShared {
    unsigned rowpos[kCvWarps];
    fx_t sum[kCvWarps];
    unsigned next;
    long long ws[kCvWarps];
};

__device__ __forceinline__ void cv_sync(int NW, int bar) {
    if (NW == 1)
        __syncwarp();
    else
        asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(NW * 32) : "memory");
}

// Sum over the block, in every thread.
__device__ __forceinline__ long long cv_block_sum(long long v, ConvShared &sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh.ws[threadIdx.x >> 5] = v;
    __syncthreads();
    long long t = 0;
#pragma unroll
    for (int q = 0; q < kCvWarps; q++) t += sh.ws[q];
    return t;
}

// Exclusive scan over the block; tot: the block's sum.
__device__ __forceinline__ long long cv_block_scan(long long v, ConvShared &sh, long long &tot) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    long long x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();
    if (lane == 31) sh.ws[w] = x;
    __syncthreads();
    long long pre = x - v;
    tot = 0;
#pragma unroll
    for (int q = 0; q < kCvWarps; q++) {
        if (q < w) pre += sh.ws[q];
        tot += sh.ws[q];
    }
    return pre;
}

// Sum of the other blocks' values before this block (blk[2 b + k]), and of all.
__device__ __forceinline__ long long cv_before(const int64_t *blk, int k, ConvShared &sh, long long &all) {
    long long b = 0, t = 0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += kCvT) {
        const long long c = __ldcg(blk + 2 * i + k);
        t += c;
        if (i < (int)blockIdx.x) b += c;
    }
    all = cv_block_sum(t, sh);
    return cv_block_sum(b, sh);
}

// Sums the gathered links of group g by destination (a team of NW warps, table
// slice from slot tab on) into a row at the start of its room in rk / rq; every
// entry's place in its column replaces the links in sk, so that writing the
// columns takes no second atomic.
// Keys are taken in rounds of a power of two parts of their hash so that a
// round's distinct keys fit; false if a list overflows all the same.
__device__ __forceinline__ bool sum_group(const ConvDev &a, int NW, int32_t g, int tab, ConvShared &sh) {
    const int w = threadIdx.x >> 5, w0 = w & ~(NW - 1), lane = threadIdx.x & 31, rank = threadIdx.x - w0 * 32;
    const int NT = NW * 32, bar = NW == 16 ? 5 : 1 + (w0 >> 2);
    const int mask = NW * kCvWarpTab - 1;
    const unsigned b0 = a.gloff[g], len = a.gcross[g];
    unsigned R = 1;
    if (len > (unsigned)kCvBlockMax)
        while (R * (kCvBlockMax / 2) < len) R <<= 1;
    fx_t total = 0;
    bool ok = true;
    if (rank == 0) sh.rowpos[w0] = 0;
    for (unsigned r = 0; r < R; r++) {
        int cnt = 0;
        for (unsigned j0 = 0; j0 < len; j0 += kCvIlp * NT) {
            int32_t key[kCvIlp];
            fx_t q[kCvIlp];
#pragma unroll
            for (int k = 0; k < kCvIlp; k++) {
                const unsigned j = j0 + k * NT + rank;
                key[k] = -1;
                q[k] = 0;
                if (j < len) {
                    key[k] = a.sk[b0 + j];
                    q[k] = a.sq[b0 + j];
                    if (R > 1 && ((mix32((uint32_t)key[k] ^ 0x5bd1e995u) >> 7) & (R - 1)) != r) key[k] = -1;
                }
            }
#pragma unroll
            for (int k = 0; k < kCvIlp; k++) {
                bool fresh = false;
                int s = 0;
                if (key[k] >= 0) {
                    s = tab_slot(key[k], mask);
                    int32_t prev = atomicCAS(&cv_key(tab + s), kEmpty, key[k]);
                    int probe = 0;
                    for (; prev != kEmpty && prev != key[k] && probe < mask; probe++) {
                        s = (s + 1) & mask;
                        prev = atomicCAS(&cv_key(tab + s), kEmpty, key[k]);
                    }
                    fresh = prev == kEmpty;
                    const unsigned ql = (unsigned)q[k];
                    const unsigned old = atomicAdd(&cv_lo(tab + s), ql);
                    atomicAdd(&cv_hi(tab + s),
                              (unsigned)((unsigned long long)q[k] >> 32) + (old + ql < old ? 1u : 0u));
                }
                const unsigned bal = __ballot_sync(kFull, fresh);
                const int pos = cnt + __popc(bal & ((1u << lane) - 1u));
                if (fresh && pos < kCvList) cv_list(pos) = (uint16_t)s;
                cnt += __popc(bal);
            }
        }
        // Only possible in rounds: the entries past the list, and the table with them, are dropped with the launch.
        // What is counted into the row is what is written to it, since the row is read back below.
        if (cnt > kCvList) {
            ok = false;
            cnt = kCvList;
        }
        cv_sync(NW, bar);
        unsigned pos = 0;
        if (lane == 0) pos = atomicAdd(&sh.rowpos[w0], (unsigned)cnt);
        pos = __shfl_sync(kFull, pos, 0);
        for (int q = lane; q < cnt; q += 32) {
            const int s = tab + cv_list(q);
            const int32_t k = cv_key(s);
            const fx_t v = (fx_t)(((unsigned long long)cv_hi(s) << 32) | cv_lo(s));
            cv_key(s) = kEmpty;
            cv_lo(s) = 0;
            cv_hi(s) = 0;
            a.rk[b0 + pos + q] = k;
            a.rq[b0 + pos + q] = v;
            if (R == 1) a.sk[b0 + pos + q] = (int32_t)atomicAdd(a.colcnt + k, 1u);  // every gathered link has been read
            total += v;
        }
        cv_sync(NW, bar);
    }
    if (a.sub) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(kFull, total, o);
        if (lane == 0 && total) atomic_add_fx(&a.attr[g].OUT, total);
    }
    const unsigned row = sh.rowpos[w0];
    if (rank == 0) a.rowlen[g] = row;
    if (R > 1)  // rk is the team's own writing, ordered by cv_sync
        for (unsigned j = rank; j < row; j += NT) a.sk[b0 + j] = (int32_t)atomicAdd(a.colcnt + a.rk[b0 + j], 1u);
    cv_sync(NW, bar);
    return ok;
}

__global__ void __launch_bounds__(kCvT, kCvBlocks) k_convert(const __grid_constant__ ConvDev a) {
    cg::grid_group grid = cg::this_grid();
    __shared__ ConvShared sh;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nb = (int)gridDim.x, bx = (int)blockIdx.x;
    const int64_t gtid = (int64_t)bx * kCvT + threadIdx.x, gthreads = (int64_t)nb * kCvT;
    const int64_t gw = (int64_t)w * nb + bx, nw = (int64_t)nb * kCvWarps;
    for (int s = threadIdx.x; s < kCvTab; s += kCvT) {
        cv_key(s) = kEmpty;
        cv_lo(s) = 0;
        cv_hi(s) = 0;
    }
    for (int64_t i = gtid; i < a.N; i += gthreads) {
        a.count[i] = 0;
        a.gcap[i] = a.gcross[i] = a.rowlen[i] = a.colcnt[i] = 0;
    }
    grid.sync();
    for (int64_t v = gtid; v < a.N; v += gthreads) atomicAdd(a.count + a.unit_mod[v], 1);
    grid.sync();
    // super-nodes: the non-empty modules in ascending order, a run of ids per block
    const int64_t chunk = (((int64_t)a.N + nb - 1) / nb + kCvT - 1) / kCvT * kCvT;
    const int64_t c0 = min((int64_t)a.N, bx * chunk), c1 = min((int64_t)a.N, c0 + chunk);
    long long ngl;
    {
        long long c = 0;
        for (int64_t m = c0 + threadIdx.x; m < c1; m += kCvT) c += a.count[m] > 0;
        c = cv_block_sum(c, sh);
        if (threadIdx.x == 0) a.blk[2 * bx] = c;
        grid.sync();
        long long pos = cv_before(a.blk, 0, sh, ngl);
        for (int64_t m0 = c0; m0 < c1; m0 += kCvT) {
            const int64_t m = m0 + threadIdx.x;
            const int32_t cm = m < c1 ? a.count[m] : 0;
            long long tot;
            const long long s = pos + cv_block_scan(cm > 0 ? 1 : 0, sh, tot);
            pos += tot;
            if (cm > 0) {
                a.snid[m] = (int32_t)s;
                Stat4 st = a.stat[m];
                if (a.sub) st.OUT = 0;  // a sub-module's out-flow counts all links, not its sub-problem's alone
                a.attr[s] = st;
                a.nnodes[s] = cm;
                a.mod[s] = a.sub ? a.minst[m] : (int32_t)m;
                if (a.K > 1) a.inst[s] = a.sub ? a.parent_inst[a.minst[m]] : a.minst[m];
                if (!a.sub) a.count[m] = 1;  // units of the new level in the module
            }
        }
    }
    const int32_t ng = (int32_t)ngl;
    grid.sync();
    // groups of the rows, and the most links each group can gather
    for (int64_t v = gtid; v < a.N; v += gthreads) {
        const int32_t g = a.snid[a.unit_mod[v]];
        a.node_sn[v] = g;
        if (!a.row_mod) {
            const unsigned d = (unsigned)(a.off[v + 1] - a.off[v]);
            if (d) atomicAdd(a.gcap + g, d);
        }
    }
    if (a.row_mod)
        for (int64_t u = gtid; u < a.n; u += gthreads) {
            const int32_t g = a.snid[a.row_mod[u]];
            a.group[u] = g;
            const unsigned d = (unsigned)(a.off[u + 1] - a.off[u]);
            if (d) atomicAdd(a.gcap + g, d);
        }
    grid.sync();
    const int32_t *const group = a.row_mod ? a.group : a.node_sn;
    for (int64_t g0 = gw * 32; g0 < ng; g0 += nw * 32) {  // room per group, in no particular order
        const int64_t g = g0 + lane;
        const unsigned c = g < ng ? a.gcap[g] : 0u;
        unsigned x = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(kFull, x, o);
            if (lane >= o) x += y;
        }
        unsigned base = 0;
        if (lane == 31) base = (unsigned)atomicAdd(a.ctl + 11, (unsigned long long)x);
        base = __shfl_sync(kFull, base, 31);
        if (g < ng) a.gloff[g] = base + x - c;
    }
    grid.sync();
    // links between groups, gathered into the source group's room, four per lane at a time
    for (int64_t e0 = gw * 32; e0 < a.m; e0 += nw * 32 * kCvIlp) {
        int32_t g[kCvIlp], b[kCvIlp];
        fx_t q[kCvIlp];
#pragma unroll
        for (int k = 0; k < kCvIlp; k++) {
            const int64_t e = e0 + k * nw * 32 + lane;
            g[k] = b[k] = 0;
            q[k] = 0;
            if (e0 + k * nw * 32 < a.m) {  // warp-uniform; lanes past the links read the last one
                const int64_t c = min(e, a.m - 1);
                g[k] = a.src[c];
                b[k] = a.dst[c];
                q[k] = a.fx[c];
            }
        }
#pragma unroll
        for (int k = 0; k < kCvIlp; k++) {
            g[k] = group[g[k]];
            b[k] = group[b[k]];
        }
        unsigned base[kCvIlp];
        int head[kCvIlp];
#pragma unroll
        for (int k = 0; k < kCvIlp; k++) {
            if (e0 + k * nw * 32 + lane >= a.m || b[k] == g[k]) g[k] = -1;
            // lanes of a run of links with the same source group (rows follow one another) take their places together
            const int32_t before = __shfl_up_sync(kFull, g[k], 1);
            const unsigned heads = __ballot_sync(kFull, lane == 0 || before != g[k]);
            head[k] = 31 - __clz(heads & (kFull >> (31 - lane)));
            const unsigned after = lane == 31 ? 0u : heads & (kFull << (lane + 1));
            const int end = after ? __ffs(after) - 1 : 32;
            base[k] = 0;
            if (g[k] >= 0 && lane == head[k]) base[k] = atomicAdd(a.gcross + g[k], (unsigned)(end - head[k]));
        }
#pragma unroll
        for (int k = 0; k < kCvIlp; k++) {
            base[k] = __shfl_sync(kFull, base[k], head[k]);
            if (g[k] >= 0) {
                const unsigned p = a.gloff[g[k]] + base[k] + (unsigned)(lane - head[k]);
                a.sk[p] = b[k];
                a.sq[p] = q[k];
            }
        }
    }
    grid.sync();
    // groups by team size
    for (int64_t g0 = gw * 32; g0 < ng; g0 += nw * 32) {
        const int64_t g = g0 + lane;
        const unsigned l = g < ng ? a.gcross[g] : 0u;
        const int c = l == 0 ? -1 : l <= (unsigned)kCvWarpMax ? 0 : l <= (unsigned)kCvTeamMax ? 1 : 2;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const unsigned bal = __ballot_sync(kFull, c == k);
            unsigned base = 0;
            if (bal && lane == 0) base = (unsigned)atomicAdd(a.ctl + 8 + k, (unsigned long long)__popc(bal));
            base = __shfl_sync(kFull, base, 0);
            if (c == k) a.list[(int64_t)k * a.N + base + __popc(bal & ((1u << lane) - 1u))] = (int32_t)g;
        }
        if (__any_sync(kFull, l > (unsigned)kCvMost) && lane == 0) a.ctl[2] = 1;
    }
    grid.sync();
    if (__ldcg(a.ctl + 2)) return;  // the same in every block
    {
        const int n0 = (int)__ldcg(a.ctl + 8), n1 = (int)__ldcg(a.ctl + 9), n2 = (int)__ldcg(a.ctl + 10);
        bool ok = true;
        int phase = n2 > 0 ? 0 : 1;
        int64_t i = 0;
        for (;;) {
            int NW, g;
            if (phase == 0) {
                __syncthreads();
                if (threadIdx.x == 0) sh.next = (unsigned)atomicAdd(a.ctl + 12, 1ull);
                __syncthreads();
                if (sh.next >= (unsigned)n2) {
                    phase = 1;
                    i = 0;
                    __syncthreads();
                    continue;
                }
                NW = 16;
                g = a.list[(int64_t)2 * a.N + sh.next];
            } else if (phase == 1) {
                const int64_t k = (w >> 2) * (int64_t)nb + bx + i * 4 * nb;
                i++;
                if (k >= n1) {
                    phase = 2;
                    i = 0;
                    continue;
                }
                NW = 4;
                g = a.list[(int64_t)a.N + k];
            } else {
                const int64_t k = gw + i * nw;
                i++;
                if (k >= n0) break;
                NW = 1;
                g = a.list[k];
            }
            ok &= sum_group(a, NW, g, (w & ~(NW - 1)) * kCvWarpTab, sh);
        }
        if (!ok) a.ctl[13] = 1;
    }
    grid.sync();
    if (__ldcg(a.ctl + 13)) return;  // the same in every block
    // CSR and CSC offsets; what the level's hub units need
    const int64_t gchunk = (((int64_t)ng + nb - 1) / nb + kCvT - 1) / kCvT * kCvT;
    const int64_t g0 = min((int64_t)ng, bx * gchunk), g1 = min((int64_t)ng, g0 + gchunk);
    {
        long long r = 0, c = 0;
        for (int64_t g = g0 + threadIdx.x; g < g1; g += kCvT) {
            r += a.rowlen[g];
            c += a.colcnt[g];
        }
        r = cv_block_sum(r, sh);
        c = cv_block_sum(c, sh);
        if (threadIdx.x == 0) {
            a.blk[2 * bx] = r;
            a.blk[2 * bx + 1] = c;
        }
        grid.sync();
        long long mr, mc;
        long long pr = cv_before(a.blk, 0, sh, mr), pc = cv_before(a.blk, 1, sh, mc);
        for (int64_t q0 = g0; q0 < g1; q0 += kCvT) {
            const int64_t g = q0 + threadIdx.x;
            const long long rl = g < g1 ? a.rowlen[g] : 0, cl = g < g1 ? a.colcnt[g] : 0;
            long long tr, tc;
            const long long er = cv_block_scan(rl, sh, tr), ec = cv_block_scan(cl, sh, tc);
            if (g < g1) {
                a.out_off[g] = pr + er;
                a.in_off[g] = pc + ec;
                const long long d = rl + cl;
                if (d > a.hub_bound) {
                    atomicAdd(a.ctl + 3, 1ull);
                    atomicAdd(a.ctl + 4, (unsigned long long)min(a.hub_max_parts, (int64_t)((d + a.hub_part - 1) / a.hub_part)));
                    atomicAdd(a.ctl + 5, (unsigned long long)d);
                    atomicAdd(a.ctl + 6, (unsigned long long)((d + a.hub_chunk - 1) / a.hub_chunk));
                }
            }
            pr += tr;
            pc += tc;
        }
        if (bx == 0 && threadIdx.x == 0) {
            a.out_off[ng] = mr;
            a.in_off[ng] = mc;
            a.ctl[0] = (unsigned long long)ng;
            a.ctl[1] = (unsigned long long)mr;
        }
    }
    grid.sync();
    // rows, eight lanes each (the whole warp for rows of more than 64 entries), and their entries in the columns
    auto put = [&](int32_t g, unsigned from, int64_t to, unsigned len, int r, int width) {
        for (unsigned j0 = 0; j0 < len; j0 += kCvIlp * width) {
            int32_t b[kCvIlp], at[kCvIlp];
            fx_t q[kCvIlp];
            int64_t p[kCvIlp];
#pragma unroll
            for (int k = 0; k < kCvIlp; k++) {
                const unsigned j = j0 + k * width + r;
                b[k] = -1;
                if (j < len) {
                    b[k] = a.rk[from + j];
                    at[k] = a.sk[from + j];
                    q[k] = a.rq[from + j];
                }
            }
#pragma unroll
            for (int k = 0; k < kCvIlp; k++)
                if (b[k] >= 0) p[k] = a.in_off[b[k]] + at[k];
#pragma unroll
            for (int k = 0; k < kCvIlp; k++)
                if (b[k] >= 0) {
                    const int64_t j = to + j0 + k * width + r;
                    a.out_dst[j] = b[k];
                    a.out_fx[j] = q[k];
                    a.out_src[j] = g;
                    a.in_src[p[k]] = g;
                    a.in_fx[p[k]] = q[k];
                }
        }
    };
    for (int64_t r0 = gw * 4; r0 < ng; r0 += nw * 4) {
        const int64_t g = r0 + (lane >> 3);
        const unsigned from = g < ng ? a.gloff[g] : 0u, len = g < ng ? a.rowlen[g] : 0u;
        const int64_t to = g < ng ? a.out_off[g] : 0;
        if (len <= 64) put((int32_t)g, from, to, len, lane & 7, 8);
        __syncwarp();
        for (int k = 0; k < 4; k++) {
            const unsigned l = __shfl_sync(kFull, len, 8 * k);
            if (l > 64)
                put((int32_t)(r0 + k), __shfl_sync(kFull, from, 8 * k), __shfl_sync(kFull, to, 8 * k), l, lane, 32);
        }
    }
}

}  // namespace

bool convert_fused(const ConvertArgs &c, ConvertResult &out, Arena &ar, cudaStream_t s) {
    static std::mutex mu;
    static std::vector<int> resident;  // per device
    int dev = 0;
    RMX_CUDA(cudaGetDevice(&dev));
    {
        std::lock_guard<std::mutex> lk(mu);
        if ((int)resident.size() <= dev) resident.resize(dev + 1, 0);
        if (resident[dev] == 0) {
            RMX_CUDA(cudaFuncSetAttribute(k_convert, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCvSmem));
            RMX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident[dev], k_convert, kCvT, kCvSmem));
        }
        if (resident[dev] < 1) throw CudaError(cudaErrorLaunchOutOfResources, "conversion kernel does not fit an SM");
    }
    const size_t mk = ar.mark();
    const int32_t N = c.N;
    const int64_t m = std::max<int64_t>(c.m, 1);
    if (ar.cap - ar.mark() < (size_t)m * 24 + (size_t)N * 36 + (size_t)c.src->n * 4 + (1 << 16))
        return false;  // far more nodes than links: the other path needs less scratch
    const int nb = (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)std::min(resident[dev], kCvBlocks) * num_sms(), std::max<int64_t>(m / 2048, N / 512)));
    ConvDev a;
    a.N = N;
    a.unit_mod = c.unit_mod;
    a.count = c.M->count;
    a.stat = c.M->stat;
    a.minst = c.M->inst;
    a.parent_inst = c.parent_inst;
    a.sub = c.sub ? 1 : 0;
    a.K = c.K;
    a.n = c.src->n;
    a.m = c.m;
    a.off = c.src->out_off;
    a.dst = c.src->out_dst;
    a.src = c.src->out_src;
    a.fx = c.src->out_fx;
    a.row_mod = c.row_mod;
    a.mod = c.dst->mod;
    a.nnodes = c.dst->nnodes;
    a.inst = c.dst->inst;
    a.node_sn = c.node_sn;
    a.attr = c.dst->attr;
    a.out_off = c.dst->out_off;
    a.in_off = c.dst->in_off;
    a.out_dst = c.dst->out_dst;
    a.out_src = c.dst->out_src;
    a.in_src = c.dst->in_src;
    a.out_fx = c.dst->out_fx;
    a.in_fx = c.dst->in_fx;
    a.snid = ar.alloc<int32_t>(N);
    a.group = c.row_mod ? ar.alloc<int32_t>(std::max(c.src->n, 1)) : nullptr;
    a.gcap = ar.alloc<unsigned>(N);
    a.gloff = ar.alloc<unsigned>(N);
    a.gcross = ar.alloc<unsigned>(N);
    a.rowlen = ar.alloc<unsigned>(N);
    a.colcnt = ar.alloc<unsigned>(N);
    a.sk = ar.alloc<int32_t>(m);
    a.sq = ar.alloc<fx_t>(m);
    a.rk = ar.alloc<int32_t>(m);
    a.rq = ar.alloc<fx_t>(m);
    a.list = ar.alloc<int32_t>(3 * (size_t)N);
    a.blk = ar.alloc<int64_t>(2 * (size_t)nb);
    a.ctl = ar.alloc<unsigned long long>(16);
    a.hub_bound = c.hub.bound;
    a.hub_part = c.hub.part;
    a.hub_chunk = c.hub.chunk;
    a.hub_max_parts = c.hub.max_parts;
    RMX_CUDA(cudaMemsetAsync(a.ctl, 0, sizeof(unsigned long long) * 16, s));
    void *args[] = {(void *)&a};
    RMX_CUDA(cudaLaunchCooperativeKernel((void *)k_convert, dim3(nb), dim3(kCvT), args, kCvSmem, s));
    RMX_LAUNCHED();
    unsigned long long r[14];
    RMX_CUDA(cudaMemcpyAsync(r, a.ctl, sizeof r, cudaMemcpyDeviceToHost, s));
    RMX_CUDA(cudaStreamSynchronize(s));
    ar.release(mk);
    if (r[2] || r[13]) return false;
    out.n = (int32_t)r[0];
    out.m = (int64_t)r[1];
    for (int k = 0; k < 4; k++) out.hub[k] = (int64_t)r[3 + k];
    return true;
}

}  // namespace rmx

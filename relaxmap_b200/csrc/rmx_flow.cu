// Graph construction and stationary flow.
//
// build_csr     loader edge map + edge preparation (FileIO.cpp:157, :220;
//               OmpRelaxmap.cpp:117-135, 158-162) as a stable radix sort of
//               (src,dst), sequential in-order duplicate sums, compaction, and
//               a stable transpose for the in-links.
// normalise     Network::initiate's dangling detection and row normalisation
//               (Module.cpp:228-247), sequential row sums as in the reference.
// power_iteration  calculateSteadyState (Module.cpp:340-469) as ONE cooperative
//               persistent launch: pull SpMV over the CSC with the teleport and
//               dangling terms folded in, deterministic grid reductions for the
//               normaliser, L1 change and dangling mass, the reference's stop
//               rule evaluated identically by every block.
// edge_flows    Module.cpp:275-286 plus the fixed-point unit attributes.
#include <cooperative_groups.h>

#include <algorithm>
#include <climits>
#include <mutex>
#include <vector>

#include "rmx_engine.cuh"

namespace cg = cooperative_groups;

namespace rmx {

constexpr unsigned kFull = 0xffffffffu;

static int bits_for(int64_t n) {
    int b = 1;
    while ((int64_t(1) << b) < n) b++;
    return b;
}

// ------------------------------------------------------------ CSR build

__global__ void k_make_keys(const int32_t *src, const int32_t *dst, int64_t n, int b, uint64_t *keys, uint32_t *vals) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
        keys[e] = ((uint64_t)(uint32_t)src[e] << b) | (uint32_t)dst[e];
        vals[e] = (uint32_t)e;
    }
}

__global__ void k_heads(const uint64_t *keys, int64_t n, uint8_t *flag) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
        flag[e] = (e == 0 || keys[e] != keys[e - 1]) ? 1 : 0;
}

// One thread per distinct (src,dst): weights summed sequentially in input order.
__global__ void k_sum_dups(const uint64_t *keys, const uint32_t *vals, const double *w, const int32_t *head,
                           const int64_t *n_heads, int64_t n, int b, int32_t *usrc, int32_t *udst, double *uw,
                           uint8_t *keep, unsigned long long *n_self) {
    int64_t U = *n_heads;
    uint64_t mask = (uint64_t(1) << b) - 1;
    for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < U; u += (int64_t)gridDim.x * blockDim.x) {
        int64_t beg = head[u], end = (u + 1 < U) ? head[u + 1] : n;
        double s = w[vals[beg]];
        for (int64_t j = beg + 1; j < end; j++) s += w[vals[j]];
        uint64_t k = keys[beg];
        int32_t a = (int32_t)(k >> b), d = (int32_t)(k & mask);
        usrc[u] = a;
        udst[u] = d;
        uw[u] = s;
        bool pos = s > 0.0;
        keep[u] = (pos && a != d) ? 1 : 0;
        if (pos && a == d) atomicAdd(n_self, 1ull);
    }
}

__global__ void k_gather_kept(const int32_t *kept, const int64_t *n_kept, const int32_t *usrc, const int32_t *udst,
                              const double *uw, int32_t *lsrc, int32_t *out_dst, double *out_w0,
                              unsigned long long *row_count) {
    int64_t K = *n_kept;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < K; i += (int64_t)gridDim.x * blockDim.x) {
        int32_t u = kept[i];
        lsrc[i] = usrc[u];
        out_dst[i] = udst[u];
        out_w0[i] = uw[u];
        atomicAdd(&row_count[usrc[u]], 1ull);
    }
}

__global__ void k_dst_keys(const int32_t *dst, int64_t m, uint64_t *keys, uint32_t *vals, unsigned long long *col_count) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        keys[i] = (uint64_t)(uint32_t)dst[i];
        vals[i] = (uint32_t)i;
        atomicAdd(&col_count[dst[i]], 1ull);
    }
}

__global__ void k_gather_csc(const uint32_t *perm, int64_t m, const int32_t *lsrc, const double *w0, int32_t *in_src,
                             double *in_w) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t j = perm[i];
        in_src[i] = lsrc[j];
        in_w[i] = w0[j];
    }
}

CsrBuild build_csr(int32_t n, int64_t n_edges, int32_t *d_src, int32_t *d_dst, double *d_w, int64_t *out_off,
                   int32_t *out_dst, double *out_w0, int64_t *in_off, int32_t *in_src, double *in_w, Arena &ar,
                   cudaStream_t s, int64_t *scratch_dev) {
    CsrBuild r;
    const int T = 256;
    const unsigned G = (unsigned)std::max<int64_t>(1, std::min<int64_t>((n_edges + T - 1) / T, num_sms() * 32));
    RMX_CUDA(cudaMemsetAsync(out_off, 0, sizeof(int64_t) * (n + 1), s));
    RMX_CUDA(cudaMemsetAsync(in_off, 0, sizeof(int64_t) * (n + 1), s));
    if (n_edges == 0) return r;
    size_t mk = ar.mark();
    const int b = bits_for(std::max<int64_t>(n, 2));
    uint64_t *keys = ar.alloc<uint64_t>(n_edges), *keys2 = ar.alloc<uint64_t>(n_edges);
    uint32_t *vals = ar.alloc<uint32_t>(n_edges), *vals2 = ar.alloc<uint32_t>(n_edges);
    k_make_keys<<<G, T, 0, s>>>(d_src, d_dst, n_edges, b, keys, vals);
    RMX_LAUNCHED();
    radix_sort_pairs(keys, vals, keys2, vals2, n_edges, 2 * b, ar, s);
    uint8_t *flag = ar.alloc<uint8_t>(n_edges);
    k_heads<<<G, T, 0, s>>>(keys, n_edges, flag);
    RMX_LAUNCHED();
    int32_t *head = ar.alloc<int32_t>(n_edges);
    int64_t *cnt = scratch_dev;  // [0] heads [1] kept [2] self-loops
    RMX_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int64_t) * 3, s));
    compact_flags(flag, n_edges, head, cnt + 0, ar, s);
    int32_t *usrc = ar.alloc<int32_t>(n_edges), *udst = ar.alloc<int32_t>(n_edges);
    double *uw = ar.alloc<double>(n_edges);
    uint8_t *keep = flag;  // reuse
    k_sum_dups<<<G, T, 0, s>>>(keys, vals, d_w, head, cnt + 0, n_edges, b, usrc, udst, uw, keep,
                               reinterpret_cast<unsigned long long *>(cnt + 2));
    RMX_LAUNCHED();
    int64_t U = 0;
    RMX_CUDA(cudaMemcpyAsync(&U, cnt + 0, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    RMX_CUDA(cudaStreamSynchronize(s));
    int32_t *kept = ar.alloc<int32_t>(std::max<int64_t>(U, 1));
    compact_flags(keep, U, kept, cnt + 1, ar, s);
    int32_t *lsrc = ar.alloc<int32_t>(std::max<int64_t>(U, 1));
    k_gather_kept<<<G, T, 0, s>>>(kept, cnt + 1, usrc, udst, uw, lsrc, out_dst, out_w0,
                                  reinterpret_cast<unsigned long long *>(out_off));
    RMX_LAUNCHED();
    int64_t host_cnt[3];
    RMX_CUDA(cudaMemcpyAsync(host_cnt, cnt, sizeof(host_cnt), cudaMemcpyDeviceToHost, s));
    RMX_CUDA(cudaStreamSynchronize(s));
    const int64_t m = host_cnt[1];
    r.n_links = m;
    r.n_self = host_cnt[2];
    scan_exclusive(out_off, out_off, n + 1, nullptr, ar, s);
    if (m > 0) {
        k_dst_keys<<<G, T, 0, s>>>(out_dst, m, keys, vals, reinterpret_cast<unsigned long long *>(in_off));
        RMX_LAUNCHED();
        radix_sort_pairs(keys, vals, keys2, vals2, m, b, ar, s);
        k_gather_csc<<<G, T, 0, s>>>(vals, m, lsrc, out_w0, in_src, in_w);
        RMX_LAUNCHED();
    }
    scan_exclusive(in_off, in_off, n + 1, nullptr, ar, s);
    ar.release(mk);
    return r;
}

// ------------------------------------------------------------ normalise

// Per-row kernels take 32 consecutive rows per warp: a lane handles a row of
// up to kRowSeqMax links by itself, in link order (the reference's order);
// heavier rows (R-MAT hubs reach 10^5-10^6 links) are then taken by the whole
// warp one at a time, lanes striding the links, so that no lane walks a hub
// while the rest of the grid has finished.
constexpr int64_t kRowSeqMax = 256;

// Sum over the warp in a fixed butterfly order: every lane gets the same value.
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

// Row sums and normalised weights (Module.cpp:237-247: sum of the out-link
// weights in link order, then each weight divided by it; a heavy row's sum is
// formed by the warp, which rounds differently in the last bits).
__global__ void k_normalise_rows(int32_t n, const int64_t *off, const double *w0, double *wn, double *rowsum,
                                 uint8_t *dangling) {
    const int lane = threadIdx.x & 31;
    const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t base = gw * 32; base < n; base += nw * 32) {
        const int64_t i = base + lane;
        bool heavy = false;
        if (i < n) {
            const int64_t b = off[i], e = off[i + 1];
            heavy = e - b > kRowSeqMax;
            if (!heavy) {
                double s = 0.0;
                for (int64_t j = b; j < e; j++) s += w0[j];
                for (int64_t j = b; j < e; j++) wn[j] = w0[j] / s;
                rowsum[i] = s;
            }
            dangling[i] = (b == e) ? 1 : 0;
        }
        for (unsigned hv = __ballot_sync(kFull, heavy); hv; hv &= hv - 1) {
            const int64_t r = base + __ffs(hv) - 1;
            const int64_t b = off[r], e = off[r + 1];
            double s = 0.0;
            for (int64_t j = b + lane; j < e; j += 32) s += w0[j];
            s = warp_sum(s);
            for (int64_t j = b + lane; j < e; j += 32) wn[j] = w0[j] / s;
            if (lane == 0) rowsum[r] = s;
        }
    }
}

__global__ void k_normalise_cols(int64_t m, const int32_t *in_src, const double *raw, double *wn,
                                 const double *rowsum) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x)
        wn[k] = raw[k] / rowsum[in_src[k]];
}

void normalise(int32_t n, const int64_t *out_off, const double *out_w0, double *out_f, const int64_t *in_off,
               const int32_t *in_src, const double *in_w_raw, double *in_w, uint8_t *dangling, Arena &ar,
               cudaStream_t s, bool cols) {
    size_t mk = ar.mark();
    double *rowsum = ar.alloc<double>(std::max(n, 1));
    k_normalise_rows<<<blocks_for(n, 256, num_sms() * 32), 256, 0, s>>>(n, out_off, out_w0, out_f, rowsum, dangling);
    RMX_LAUNCHED();
    int64_t m = 0;
    if (cols) {
        RMX_CUDA(cudaMemcpyAsync(&m, in_off + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
        RMX_CUDA(cudaStreamSynchronize(s));
    }
    if (m > 0) {
        k_normalise_cols<<<blocks_for(m, 256, num_sms() * 32), 256, 0, s>>>(m, in_src, in_w_raw, in_w, rowsum);
        RMX_LAUNCHED();
    }
    ar.release(mk);
}

// ------------------------------------------------------------ power iteration

template <int NT>
__device__ __forceinline__ double block_sum(double v, double *sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sh[w] = v;
    __syncthreads();
    double t = 0.0;
    if (w == 0) {
        t = lane < NT / 32 ? sh[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(kFull, t, o);
    }
    __syncthreads();
    return t;  // valid in thread 0
}

// Sum of nb per-block partials in one fixed order (lane-strided, then a
// butterfly), by the calling warp; loads run eight ahead of the additions.
__device__ __forceinline__ double warp_sum_parts(const double *parts, int nb, int lane) {
    double v = 0.0;
    for (int i0 = lane; i0 < nb; i0 += 256) {
        double t[8];
#pragma unroll
        for (int k = 0; k < 8; k++) t[k] = i0 + 32 * k < nb ? __ldcg(parts + i0 + 32 * k) : 0.0;
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (i0 + 32 * k < nb) v += t[k];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

// warp_sum_parts over shared memory.
__device__ __forceinline__ double shared_sum_parts(const double *parts, int nb, int lane) {
    double v = 0.0;
#pragma unroll 4
    for (int i = lane; i < nb; i += 32) v += parts[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

constexpr int kPowT = 256;

// out[k] = the sum of parts[k] as warp_sum_parts forms it, in every thread of the
// block (K = 1 or 2). FEW: at most kPowFew partial sums, as many as two blocks per
// SM; a thread loads one of each (a warp's threads two) and the warps add from
// shared memory, one latency of L2 where a warp that loads its own 4 to 9 pays
// two. A form of k_power of its own: two blocks per SM leave room for 128
// registers, and a choice at run time took some from the pull of larger graphs
// (120,000 nodes 1016 and 976 us). 50 iterations, this form and the other: 8,192
// nodes 346 and 446 us, 12,000 nodes 364 and 479, 16,000 nodes 378 and 490,
// 18,432 nodes 377 and 423.
constexpr int kPowFew = kPowT + 32;
template <bool FEW, int K>
__device__ __forceinline__ void block_sum_parts(const double *const (&parts)[K], int nb, double *out,
                                                double (*staged)[kPowFew]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (FEW) {
        const int i = threadIdx.x, i2 = i + kPowT;
        double t[K], t2[K];
#pragma unroll
        for (int k = 0; k < K; k++) {
            if (i < nb) t[k] = __ldcg(parts[k] + i);
            if (i2 < nb) t2[k] = __ldcg(parts[k] + i2);
        }
#pragma unroll
        for (int k = 0; k < K; k++) {
            if (i < nb) staged[k][i] = t[k];
            if (i2 < nb) staged[k][i2] = t2[k];
        }
        __syncthreads();
    }
    if (warp < K) {
        const double *const p = warp == 0 ? parts[0] : parts[K - 1];
        const double v = FEW ? shared_sum_parts(staged[warp], nb, lane) : warp_sum_parts(p, nb, lane);
        if (lane == 0) out[warp] = v;
    }
    __syncthreads();
}

// The iteration's sums (total flow, L1 change, dangling mass) are formed per
// "virtual" block of kPowT threads of a fixed grid, kPowGrid such blocks per
// SM, and added in block order: their rounding, which the 1e-15 stop rule sits
// on, does not depend on how many blocks are launched or in which form.
#ifndef RMX_POW_MINB
#define RMX_POW_MINB 6
#endif
constexpr int kPowGrid = 6, kPowWarps = kPowT / 32;

// Rows of more than heavy_deg in-links (in-degree hubs) are not left to one
// lane group: their links come in chunks of kPowChunk, a warp per chunk, and
// after a grid barrier every such row sums its chunks' partials in chunk order.
constexpr int64_t kPowChunk = 256;
struct PowSplit {
    const int32_t *rows = nullptr;       // heavy rows
    int32_t n_rows = 0;
    const int64_t *row_chunk = nullptr;  // chunks of heavy row h: row_chunk[h] .. row_chunk[h+1]
    const int64_t *chunk_beg = nullptr, *chunk_end = nullptr;  // link range of every chunk
    int64_t n_chunks = 0;
    double *cpart = nullptr;             // partial pull of every chunk
    double *ls = nullptr;                // per thread of the virtual grid: its light rows' sum
    int64_t heavy_deg = INT64_MAX;
};

// The flow vector's gathered copy: on graphs whose flow vector is larger
// than about half of L2 (gather_copy has the rule) the pull gathers from a copy
// holding only the nodes that have out-links (rank[i] >= 0: node i's place in it;
// gsrc: in_src renumbered to those places), of which more stays in L2. Values are the same doubles,
// so the sums are unchanged.
struct PowGather {
    const int32_t *gsrc = nullptr;  // nullptr: gather from x itself
    const int32_t *rank = nullptr;
    double *xc = nullptr;
};

// FEW: at most kPowFew virtual blocks.
template <int VEC, bool FEW>
__global__ void __launch_bounds__(kPowT, FEW ? 2 : RMX_POW_MINB) k_power(const int64_t *__restrict__ in_off, const int32_t *__restrict__ in_src,
                                                 const double *__restrict__ in_w, const double *__restrict__ tw,
                                                 const uint8_t *__restrict__ dang, int32_t n, double *x, double *y,
                                                 double *parts, int *iters_out, double alpha, PowSplit sp,
                                                 PowGather pg, int nb) {
    cg::grid_group grid = cg::this_grid();
    __shared__ double sh[32];
    __shared__ double shared_sum[2], staged[FEW ? 2 : 1][kPowFew];
    double *Sp = parts, *Dp = parts + nb, *Ep = parts + 2 * nb;
    const int64_t gthreads = (int64_t)nb * kPowT, nwarps = gthreads >> 5;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane / VEC, lv = lane % VEC;
    constexpr int RPW = 32 / VEC;  // rows per warp step
    const double beta = 1.0 - alpha;  // 1.0 - 0.15 is kBeta exactly

    // the link arrays are streamed with the evict-first hint so that the
    // gathered vector stays in L2 between iterations
    const double *xg = pg.gsrc ? pg.xc : x;          // the vector the pull gathers from
    const int32_t *gs = pg.gsrc ? pg.gsrc : in_src;  // and the links' places in it
    const double x0 = 1.0 / n;
    for (int vb = blockIdx.x; vb < nb; vb += gridDim.x) {
        double dl = 0.0;
        for (int64_t i = (int64_t)vb * kPowT + threadIdx.x; i < n; i += gthreads) {
            x[i] = x0;
            if (pg.gsrc && pg.rank[i] >= 0) pg.xc[pg.rank[i]] = x0;
            if (dang[i]) dl += x0;
        }
        dl = block_sum<kPowT>(dl, sh);
        if (threadIdx.x == 0) Dp[vb] = dl;
    }
    grid.sync();
    block_sum_parts<FEW, 1>({Dp}, nb, shared_sum + 1, staged);
    int iter = 0;
    for (;;) {
        const double D = shared_sum[1];
        const double coef = alpha + beta * D;
        for (int vb = blockIdx.x; vb < nb; vb += gridDim.x) {
            double ls = 0.0;
            const int64_t gwarp = (int64_t)vb * kPowWarps + warp;
            for (int64_t base = gwarp * RPW; base < n; base += nwarps * RPW) {
                const int64_t r = base + sub;
                double acc = 0.0;
                bool mine = r < n;
                if (mine) {
                    const int64_t b = in_off[r], e = in_off[r + 1];
                    mine = e - b <= sp.heavy_deg;
                    if (mine)
                        for (int64_t k = b + lv; k < e; k += VEC)
                            acc += beta * __ldcs(in_w + k) * __ldcg(xg + __ldcs(gs + k));
                }
#pragma unroll
                for (int o = VEC / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
                if (mine && lv == 0) {
                    const double v = coef * tw[r] + acc;
                    y[r] = v;
                    ls += v;
                }
            }
            if (sp.n_rows > 0) {  // the same branch in every block
                for (int64_t c = gwarp; c < sp.n_chunks; c += nwarps) {
                    double acc = 0.0;
                    for (int64_t k = sp.chunk_beg[c] + lane; k < sp.chunk_end[c]; k += 32)
                        acc += beta * __ldcs(in_w + k) * __ldcg(xg + __ldcs(gs + k));
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
                    if (lane == 0) sp.cpart[c] = acc;
                }
                sp.ls[(int64_t)vb * kPowT + threadIdx.x] = ls;  // until the chunks are all there
            } else {
                ls = block_sum<kPowT>(ls, sh);
                if (threadIdx.x == 0) Sp[vb] = ls;
            }
        }
        if (sp.n_rows > 0) {
            grid.sync();
            for (int vb = blockIdx.x; vb < nb; vb += gridDim.x) {
                double ls = sp.ls[(int64_t)vb * kPowT + threadIdx.x];
                for (int64_t h = (int64_t)vb * kPowWarps + warp; h < sp.n_rows; h += nwarps) {
                    const int32_t r = sp.rows[h];
                    double acc = 0.0;
                    for (int64_t c = sp.row_chunk[h] + lane; c < sp.row_chunk[h + 1]; c += 32)
                        acc += __ldcg(sp.cpart + c);
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
                    if (lane == 0) {
                        const double v = coef * tw[r] + acc;
                        y[r] = v;
                        ls += v;
                    }
                }
                ls = block_sum<kPowT>(ls, sh);
                if (threadIdx.x == 0) Sp[vb] = ls;
            }
        }
        grid.sync();
        block_sum_parts<FEW, 1>({Sp}, nb, shared_sum, staged);
        const double S = shared_sum[0];
        for (int vb = blockIdx.x; vb < nb; vb += gridDim.x) {
            double el = 0.0, dl = 0.0;
            for (int64_t i = (int64_t)vb * kPowT + threadIdx.x; i < n; i += gthreads) {
                const double xn = __ldcg(y + i) / S;
                el += fabs(xn - x[i]);
                x[i] = xn;
                if (pg.gsrc && pg.rank[i] >= 0) pg.xc[pg.rank[i]] = xn;
                if (dang[i]) dl += xn;
            }
            el = block_sum<kPowT>(el, sh);
            dl = block_sum<kPowT>(dl, sh);
            if (threadIdx.x == 0) {
                Ep[vb] = el;
                Dp[vb] = dl;
            }
        }
        grid.sync();
        block_sum_parts<FEW, 2>({Ep, Dp}, nb, shared_sum, staged);
        const double diff = shared_sum[0];
        iter++;
        if (iter >= 200 || (diff <= 1.0e-15 && iter >= 50)) break;  // Module.cpp:460
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *iters_out = iter;
}

__global__ void k_pow_heavy_flags(int32_t n, const int64_t *in_off, int64_t heavy_deg, uint8_t *flag) {
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x)
        flag[r] = in_off[r + 1] - in_off[r] > heavy_deg ? 1 : 0;
}

__global__ void k_pow_heavy_ranges(const int32_t *rows, int64_t nh, const int64_t *in_off, int64_t *be) {
    for (int64_t h = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; h < nh; h += (int64_t)gridDim.x * blockDim.x) {
        be[2 * h] = in_off[rows[h]];
        be[2 * h + 1] = in_off[rows[h] + 1];
    }
}

// The heavy rows of a CSC and their chunk tables, in arena memory (released
// with the caller's mark).
static PowSplit heavy_split(int32_t n, const int64_t *in_off, int64_t heavy_deg, Arena &ar, cudaStream_t s) {
    PowSplit sp;
    if (n <= 0) return sp;
    uint8_t *flag = ar.alloc<uint8_t>(n);
    int32_t *rows = ar.alloc<int32_t>(n);
    int64_t *cnt = ar.alloc<int64_t>(1);
    k_pow_heavy_flags<<<blocks_for(n, 256, num_sms() * 32), 256, 0, s>>>(n, in_off, heavy_deg, flag);
    RMX_LAUNCHED();
    compact_flags(flag, n, rows, cnt, ar, s);
    int64_t nh = 0;
    RMX_CUDA(cudaMemcpyAsync(&nh, cnt, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    RMX_CUDA(cudaStreamSynchronize(s));
    if (nh == 0) return sp;
    int64_t *be = ar.alloc<int64_t>(2 * nh);
    k_pow_heavy_ranges<<<blocks_for(nh, 256, num_sms() * 8), 256, 0, s>>>(rows, nh, in_off, be);
    RMX_LAUNCHED();
    std::vector<int64_t> hbe(2 * nh);
    RMX_CUDA(cudaMemcpyAsync(hbe.data(), be, sizeof(int64_t) * 2 * nh, cudaMemcpyDeviceToHost, s));
    RMX_CUDA(cudaStreamSynchronize(s));
    std::vector<int64_t> rc(nh + 1, 0), cb, ce;
    for (int64_t h = 0; h < nh; h++) {
        for (int64_t k = hbe[2 * h]; k < hbe[2 * h + 1]; k += kPowChunk) {
            cb.push_back(k);
            ce.push_back(std::min(k + kPowChunk, hbe[2 * h + 1]));
        }
        rc[h + 1] = (int64_t)cb.size();
    }
    const int64_t nc = (int64_t)cb.size();
    int64_t *d_rc = ar.alloc<int64_t>(nh + 1), *d_cb = ar.alloc<int64_t>(nc), *d_ce = ar.alloc<int64_t>(nc);
    double *cpart = ar.alloc<double>(nc);
    RMX_CUDA(cudaMemcpyAsync(d_rc, rc.data(), sizeof(int64_t) * (nh + 1), cudaMemcpyHostToDevice, s));
    RMX_CUDA(cudaMemcpyAsync(d_cb, cb.data(), sizeof(int64_t) * nc, cudaMemcpyHostToDevice, s));
    RMX_CUDA(cudaMemcpyAsync(d_ce, ce.data(), sizeof(int64_t) * nc, cudaMemcpyHostToDevice, s));
    RMX_CUDA(cudaStreamSynchronize(s));  // the host tables are freed on return
    sp.rows = rows;
    sp.n_rows = (int32_t)nh;
    sp.row_chunk = d_rc;
    sp.chunk_beg = d_cb;
    sp.chunk_end = d_ce;
    sp.n_chunks = nc;
    sp.cpart = cpart;
    sp.heavy_deg = heavy_deg;
    return sp;
}

__global__ void k_src_flags(int64_t m, const int32_t *in_src, uint32_t *flag) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x)
        flag[in_src[k]] = 1u;  // every writer stores the same value
}

__global__ void k_src_rank(int32_t n, const uint32_t *flag, const uint32_t *pos, int32_t *rank) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        rank[i] = flag[i] ? (int32_t)pos[i] : -1;
}

__global__ void k_src_remap(int64_t m, const int32_t *in_src, const int32_t *rank, int32_t *gsrc) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x)
        gsrc[k] = rank[in_src[k]];
}

// The gathered copy (PowGather) where the flow vector is larger than half of L2
// (smaller ones mostly stay there anyway: measured slower at 2^22 nodes, the
// copy's set-up costing more than it saved) and at most three quarters of the
// nodes have out-links; otherwise none. At 2^23 nodes of an R-MAT graph the flow
// takes 88 ms without it and 86 with it for 50 iterations, 339 and 325 for 200;
// at 8.2M nodes that all have out-links finding that out costs 0.2 of 56 ms. In
// arena memory (released with the caller's mark).
static PowGather gather_copy(int32_t n, const int64_t *in_off, const int32_t *in_src, Arena &ar, cudaStream_t s) {
    PowGather pg;
    constexpr int64_t kMinNodes = (int64_t)60 << 20 >> 3;  // 60 MB of doubles
    if ((int64_t)n < kMinNodes) return pg;
    int64_t m = 0;
    RMX_CUDA(cudaMemcpyAsync(&m, in_off + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    RMX_CUDA(cudaStreamSynchronize(s));
    if (m <= 0) return pg;
    const size_t mk = ar.mark();
    uint32_t *flag = ar.alloc<uint32_t>(n), *pos = ar.alloc<uint32_t>(n + 1);
    RMX_CUDA(cudaMemsetAsync(flag, 0, sizeof(uint32_t) * n, s));
    k_src_flags<<<blocks_for(m, 256, num_sms() * 32), 256, 0, s>>>(m, in_src, flag);
    RMX_LAUNCHED();
    scan_exclusive(flag, pos, n, pos + n, ar, s);
    uint32_t cnt = 0;
    RMX_CUDA(cudaMemcpyAsync(&cnt, pos + n, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    RMX_CUDA(cudaStreamSynchronize(s));
    if ((int64_t)cnt * 4 > (int64_t)n * 3) {
        ar.release(mk);
        return pg;
    }
    int32_t *rank = ar.alloc<int32_t>(n), *gsrc = ar.alloc<int32_t>(m);
    double *xc = ar.alloc<double>(std::max<uint32_t>(cnt, 1));
    k_src_rank<<<blocks_for(n, 256, num_sms() * 32), 256, 0, s>>>(n, flag, pos, rank);
    RMX_LAUNCHED();
    k_src_remap<<<blocks_for(m, 256, num_sms() * 32), 256, 0, s>>>(m, in_src, rank, gsrc);
    RMX_LAUNCHED();
    pg.gsrc = gsrc;
    pg.rank = rank;
    pg.xc = xc;
    return pg;
}

// ------------------------------------------------ small graphs: one cluster

// The same iteration for small graphs by one thread-block cluster: the flow
// vector in every block's shared memory (a new value is stored to all of
// them), the partial sums too, and the cluster's hardware barrier (0.27 us)
// where k_power has a grid barrier (1.25 us). A virtual block of k_power is 256
// threads of a block here, with the same rows, lanes and order of additions, so
// the result is the same bit for bit. Bound by two barriers and two chains of
// dependent reductions per iteration. 50 iterations, 1003 nodes: 378 us through
// k_power, 238 us here; 3001 nodes: 397 and 290 us. Rows of more than heavy_deg
// links are left to k_power (*iters_out = -1, nothing computed).
constexpr int kClT = 1024, kClGroups = kClT / kPowT, kClMaxSize = 16;
// Largest graphs: every virtual warp has one step of rows, a block has at most 8
// to 16 virtual blocks, and above four of them (which its four groups of threads
// take at once) a node costs the cluster as much as 32 links, until its 16 SMs
// take as long per iteration as the whole grid. 50 iterations here and through
// k_power: 4000 nodes and 64,000 links (four virtual blocks a block) 337 and 375
// us; above four, 1000 and 114,000 364 and 384, 2000 and 93,000 353 and 389, 3000
// and 69,000 350 and 360, 4200 and 25,000 334 and 351; beyond the bound 3500 and
// 63,000 357 and 357, 4200 and 46,000 364 and 360, 5000 and 30,000 368 and 350,
// 6000 and 96,000 455 and 374.
constexpr int32_t kClMaxNodes = 5200, kClMaxBlocks = 128, kClMaxCost = 5200;
constexpr int64_t kClMaxLinks = 1 << 17;

__device__ __forceinline__ uint32_t cl_addr(const void *p, unsigned rank) {  // p's copy in block `rank` of the cluster
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void cl_store(const void *p, unsigned rank, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(cl_addr(p, rank)), "d"(v) : "memory");
}
__device__ __forceinline__ void cl_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int VEC>
__global__ void __launch_bounds__(kClT, 1) k_power_cluster(const int64_t *__restrict__ in_off,
                                                           const int32_t *__restrict__ in_src,
                                                           const double *__restrict__ in_w,
                                                           const double *__restrict__ tw,
                                                           const uint8_t *__restrict__ dang, int32_t n, double *p,
                                                           int *iters_out, double alpha, int nb, int64_t heavy_deg) {
    extern __shared__ __align__(16) double cl_smem[];
    double *const x = cl_smem, *const y = x + n;  // y: this block's elements, by virtual block
    unsigned C, rank;
    asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(C));
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int nbe = (n + kPowT - 1) / kPowT;  // virtual blocks with an element (one per thread)
    const int ey = (nbe + (int)C - 1) / (int)C * kPowT;
    double *const Sp = y + ey, *const Ep = Sp + nb, *const Dp = Ep + nbe;
    constexpr int kMaxOwn = kClMaxBlocks / 8;  // virtual blocks of one block, of at least eight in the cluster
    __shared__ double sh[2][kMaxOwn][kPowWarps];
    __shared__ int any_heavy;
    const int t = threadIdx.x & (kPowT - 1), grp = threadIdx.x / kPowT, w = t >> 5, lane = threadIdx.x & 31;
    const int sub = lane / VEC, lv = lane % VEC, bw = threadIdx.x >> 5;
    constexpr int RPW = 32 / VEC;
    const double beta = 1.0 - alpha;
    // Virtual block vb is number vb / C of block vb % C; group g takes numbers g, g + 4, ...
    const int own = ((int)nb - (int)rank + (int)C - 1) / (int)C, owne = (nbe - (int)rank + (int)C - 1) / (int)C;
    auto warp_total = [&](double v) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
        return v;
    };
    // The sums of cnt of this block's virtual blocks, each from its eight warps' sums in
    // block_sum's order, stored to every block: warp c to block c.
    auto send = [&](const double (*q)[kPowWarps], int cnt, double *parts) {
        for (unsigned c = bw; c < C; c += kClT / 32)
            for (int k = lane; k < cnt; k += 32)
                cl_store(parts + k * (int)C + (int)rank, c,
                         ((q[k][0] + q[k][4]) + (q[k][2] + q[k][6])) + ((q[k][1] + q[k][5]) + (q[k][3] + q[k][7])));
    };
    if (threadIdx.x == 0) any_heavy = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += kClT)
        if (in_off[i + 1] - in_off[i] > heavy_deg) any_heavy = 1;
    __syncthreads();
    if (any_heavy) {  // the same in every block; no other block's memory has been touched
        if (rank == 0 && threadIdx.x == 0) *iters_out = -1;
        return;
    }
    cl_sync();  // the blocks have all started before one stores to another's memory
    const double x0 = 1.0 / n;
    for (int i = threadIdx.x; i < n; i += kClT) x[i] = x0;
    for (int k = grp; k < owne; k += kClGroups) {
        const int i = (k * (int)C + (int)rank) * kPowT + t;
        const double s = warp_total(i < n && dang[i] ? x0 : 0.0);
        if (lane == 0) sh[1][k][w] = s;
    }
    __syncthreads();
    send(sh[1], owne, Dp);
    cl_sync();
    double D = shared_sum_parts(Dp, nbe, lane);
    int iter = 0;
    for (;;) {
        const double coef = alpha + beta * D;
#pragma unroll 2
        for (int k = grp; k < own; k += kClGroups) {
            const int r = ((k * (int)C + (int)rank) * kPowWarps + w) * RPW + sub;
            double acc = 0.0, ls = 0.0;
            if (r < n) {
                const int e = (int)in_off[r + 1];
#pragma unroll 4
                for (int j = (int)in_off[r] + lv; j < e; j += VEC) acc += beta * in_w[j] * x[in_src[j]];
            }
#pragma unroll
            for (int o = VEC / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
            if (r < n && lv == 0) {
                const double v = coef * tw[r] + acc;
                const int ve = r / kPowT;  // the element's virtual block, held by block ve % C
                cl_store(y + ve / (int)C * kPowT + r % kPowT, (unsigned)(ve % (int)C), v);
                ls = v;
            }
            ls = warp_total(ls);
            if (lane == 0) sh[0][k][w] = ls;
        }
        __syncthreads();
        send(sh[0], own, Sp);
        cl_sync();
        const double S = shared_sum_parts(Sp, nb, lane);
        for (int k = grp; k < owne; k += kClGroups) {
            const int i = (k * (int)C + (int)rank) * kPowT + t;
            double el = 0.0, dl = 0.0;
            if (i < n) {
                const double xn = y[k * kPowT + t] / S;
                el = fabs(xn - x[i]);
                if (dang[i]) dl = xn;
                for (unsigned c = 0; c < C; c++) cl_store(x + i, c, xn);
            }
            el = warp_total(el);
            dl = warp_total(dl);
            if (lane == 0) {
                sh[0][k][w] = el;
                sh[1][k][w] = dl;
            }
        }
        __syncthreads();
        send(sh[0], owne, Ep);
        send(sh[1], owne, Dp);
        cl_sync();
        const double diff = shared_sum_parts(Ep, nbe, lane);
        D = shared_sum_parts(Dp, nbe, lane);
        iter++;
        if (iter >= 200 || (diff <= 1.0e-15 && iter >= 50)) break;
    }
    for (int i = (int)rank * kClT + threadIdx.x; i < n; i += (int)C * kClT) p[i] = x[i];
    if (rank == 0 && threadIdx.x == 0) *iters_out = iter;
}

// The virtual grid's blocks for n rows.
static int power_blocks(int32_t n, int vec, int max_nb) {
    return (int)std::min<int64_t>(max_nb, std::max<int64_t>(1, ((int64_t)n * vec + kPowT - 1) / kPowT));
}

// Blocks of k_power launched for nb virtual blocks: all of them (six per SM: the
// pull wants every warp it can have), or half as many, each taking two, where a
// virtual block has one to two and a quarter steps of rows: the barriers and the
// partial sums' readers then cost more than the pull gains (50 iterations, half
// and all: 60,003 nodes of degree 16 913 and 1050 us, 120,007 nodes 1217 and
// 1309; below, 30,001 nodes 642 and 575; above, 120,007 nodes of degree 24 at 8
// lanes a row 1746 and 1486, 180,001 nodes of degree 10 2764 and 2511 us for 102).
template <int VEC, bool FEW>
static int power_launch_grid(int32_t n, int nb) {
    static std::mutex mu;
    static std::vector<int> resident;  // per device
    int dev = 0;
    RMX_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    if ((int)resident.size() <= dev) resident.resize(dev + 1, 0);
    if (resident[dev] == 0) {
        int coop = 0;
        RMX_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
        if (!coop) throw CudaError(cudaErrorNotSupported, "cooperative launch not supported");
        RMX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident[dev], k_power<VEC, FEW>, kPowT, 0));
    }
    if (resident[dev] < 1) throw CudaError(cudaErrorLaunchOutOfResources, "power iteration does not fit an SM");
    const int64_t lanes = (int64_t)n * VEC, threads = (int64_t)kPowGrid * num_sms() * kPowT;
    const bool half = lanes >= threads && 4 * lanes <= 9 * threads;
    const int res = std::min(resident[dev], half ? kPowGrid / 2 : kPowGrid) * num_sms();
    const int turns = (nb + res - 1) / res;
    return (nb + turns - 1) / turns;
}

template <int VEC, bool FEW>
static void launch_power_form(int32_t n, int nb, void **args, cudaStream_t s) {
    RMX_CUDA(cudaLaunchCooperativeKernel((void *)k_power<VEC, FEW>, dim3(power_launch_grid<VEC, FEW>(n, nb)), dim3(kPowT),
                                         args, 0, s));
    RMX_LAUNCHED();
}
template <int VEC>
static void launch_power_grid(int32_t n, int nb, void **args, cudaStream_t s) {
    if (nb <= kPowFew)
        launch_power_form<VEC, true>(n, nb, args, s);
    else
        launch_power_form<VEC, false>(n, nb, args, s);
}

// Runs the cluster form if the graph is small enough (false: it is not).
// *iters (device) is -1 if a row is heavy; then nothing was computed.
template <int VEC>
static bool launch_power_cluster(int32_t n, int64_t m, const int64_t *in_off, const int32_t *in_src, const double *in_w,
                                 const double *tw, const uint8_t *dangling, double *p, int *iters, double alpha,
                                 int nb, int64_t heavy_deg, cudaStream_t s) {
    if (n > kClMaxNodes || m > kClMaxLinks || (nb > kClGroups * kClMaxSize && n + m / 32 > kClMaxCost) ||
        nb > kClMaxBlocks || (int64_t)n * VEC > (int64_t)nb * kPowT)
        return false;
    const int nbe = (n + kPowT - 1) / kPowT;
    auto smem_for = [&](int C) {
        return sizeof(double) * ((size_t)n + (size_t)((nbe + C - 1) / C) * kPowT + nb + 2 * (size_t)nbe);
    };
    static std::mutex mu;
    static std::vector<int> size;  // per device: cluster size (0 not yet asked)
    int dev = 0, C = 0;
    RMX_CUDA(cudaGetDevice(&dev));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cfg.blockDim = dim3(kClT);
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    {
        std::lock_guard<std::mutex> lk(mu);
        if ((int)size.size() <= dev) size.resize(dev + 1, 0);
        if (size[dev] == 0) {
            const size_t most = sizeof(double) * ((size_t)kClMaxNodes + kClMaxNodes / 8 + 3 * 1024);  // smem_for's largest
            RMX_CUDA(cudaFuncSetAttribute(k_power_cluster<VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
            RMX_CUDA(cudaFuncSetAttribute(k_power_cluster<VEC>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
            for (int c = kClMaxSize; c >= 1 && size[dev] == 0; c /= 2) {  // 16 blocks where a GPC has room for them
                at[0].val.clusterDim.x = c;
                cfg.gridDim = dim3(c);
                cfg.dynamicSmemBytes = most;
                int most_clusters = 0;
                if (cudaOccupancyMaxActiveClusters(&most_clusters, k_power_cluster<VEC>, &cfg) == cudaSuccess &&
                    most_clusters > 0)
                    size[dev] = c;
            }
            (void)cudaGetLastError();
            if (size[dev] == 0) size[dev] = -1;
        }
        C = size[dev];
    }
    if (C < 8) return false;
    at[0].val.clusterDim.x = C;
    cfg.gridDim = dim3(C);
    cfg.dynamicSmemBytes = smem_for(C);
    RMX_CUDA(cudaLaunchKernelEx(&cfg, k_power_cluster<VEC>, in_off, in_src, in_w, tw, dangling, n, p, iters, alpha, nb,
                                heavy_deg));
    RMX_LAUNCHED();
    return true;
}

template <int VEC>
static int launch_power(int32_t n, int64_t m, const int64_t *in_off, const int32_t *in_src, const double *in_w,
                        const double *tw, const uint8_t *dangling, double *p, Arena &ar, cudaStream_t s, double alpha) {
    int nb = power_blocks(n, VEC, kPowGrid * num_sms());
    size_t mk = ar.mark();
    int *iters = ar.alloc<int>(1);
    int h = 0;
    if (launch_power_cluster<VEC>(n, m, in_off, in_src, in_w, tw, dangling, p, iters, alpha, nb, 64 * VEC, s)) {
        RMX_CUDA(cudaMemcpyAsync(&h, iters, sizeof(int), cudaMemcpyDeviceToHost, s));
        RMX_CUDA(cudaStreamSynchronize(s));
        if (h >= 0) {
            ar.release(mk);
            return h;
        }
    }
    double *y = ar.alloc<double>(std::max(n, 1));
    double *parts = ar.alloc<double>(3 * nb);
    PowSplit sp = heavy_split(n, in_off, 64 * VEC, ar, s);
    PowGather pg = gather_copy(n, in_off, in_src, ar, s);
    if (sp.n_rows > 0) sp.ls = ar.alloc<double>((size_t)nb * kPowT);
    void *args[] = {(void *)&in_off, (void *)&in_src, (void *)&in_w,  (void *)&tw,    (void *)&dangling, (void *)&n,
                    (void *)&p,      (void *)&y,      (void *)&parts, (void *)&iters, (void *)&alpha,    (void *)&sp,
                    (void *)&pg,     (void *)&nb};
    launch_power_grid<VEC>(n, nb, args, s);
    RMX_CUDA(cudaMemcpyAsync(&h, iters, sizeof(int), cudaMemcpyDeviceToHost, s));
    RMX_CUDA(cudaStreamSynchronize(s));
    ar.release(mk);
    return h;
}

// Launch of the same solve into caller-provided scratch: y[n], parts[3 * max_blocks],
// *iters; nothing is allocated and nothing waits on the stream.
template <int VEC>
static void launch_power_into(int32_t n, int64_t m, const int64_t *in_off, const int32_t *in_src, const double *in_w,
                              const double *tw, const uint8_t *dangling, double *p, double *y, double *parts,
                              int max_blocks, int *iters, cudaStream_t s) {
    int nb = power_blocks(n, VEC, std::min(kPowGrid * num_sms(), max_blocks));
    double alpha = kAlpha;
    // No chunked rows: in-degree hubs are pulled in one pass by their own
    // lanes (nothing beyond the caller's scratch), so on graphs with such
    // hubs the sums round differently from power_iteration's. No gathered copy.
    if (launch_power_cluster<VEC>(n, m, in_off, in_src, in_w, tw, dangling, p, iters, alpha, nb, INT64_MAX, s)) return;
    PowSplit sp;
    PowGather pg;
    void *args[] = {(void *)&in_off, (void *)&in_src, (void *)&in_w,  (void *)&tw,    (void *)&dangling, (void *)&n,
                    (void *)&p,      (void *)&y,      (void *)&parts, (void *)&iters, (void *)&alpha,    (void *)&sp,
                    (void *)&pg,     (void *)&nb};
    launch_power_grid<VEC>(n, nb, args, s);
}

void power_iteration_into(int32_t n, int64_t m, const int64_t *in_off, const int32_t *in_src, const double *in_w,
                          const double *tw, const uint8_t *dangling, double *p, double *y, double *parts,
                          int max_blocks, int *iters, cudaStream_t s, int vec) {
    if (n <= 0) return;
    switch (vec) {
        case 4: return launch_power_into<4>(n, m, in_off, in_src, in_w, tw, dangling, p, y, parts, max_blocks, iters, s);
        case 8: return launch_power_into<8>(n, m, in_off, in_src, in_w, tw, dangling, p, y, parts, max_blocks, iters, s);
        case 16:
            return launch_power_into<16>(n, m, in_off, in_src, in_w, tw, dangling, p, y, parts, max_blocks, iters, s);
        default:
            return launch_power_into<32>(n, m, in_off, in_src, in_w, tw, dangling, p, y, parts, max_blocks, iters, s);
    }
}

// ------------------------------------------------ per-component power iteration

constexpr int kCompT = 256;

// Sum over the block, returned to every thread.
__device__ __forceinline__ double comp_block_sum(double v, double *sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();  // sh free from the previous use
    if (lane == 0) sh[w] = v;
    __syncthreads();
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < kCompT / 32; k++) t += sh[k];
    return t;
}

// calculateSteadyState for many independent graphs held as one disjoint union,
// all of them iterated together by one cooperative launch, each component (node
// range [lo, hi)) with its own dangling mass, normaliser, L1 change and the
// reference's stop rule (Module.cpp:340-469). tw is normalised within every
// component. Per iteration the rows of all components are pulled by the whole
// grid (each warp a run of row groups, goff: groups before each component), then
// a block per component forms its sums and normalises. The sums are those of a
// single block of kCompT threads per component. That block also pulled its rows
// before: with 40 graphs of up to 20,000 nodes and 600,000 links the largest one
// alone took 1.04 ms per iteration, 52 ms in all.
template <int VEC>
__global__ void __launch_bounds__(kCompT, 4) k_power_union(int32_t n_comp, const int64_t *__restrict__ comp,
                                                           const int64_t *__restrict__ goff,
                                                           const int64_t *__restrict__ in_off,
                                                           const int32_t *__restrict__ in_src,
                                                           const double *__restrict__ in_w,
                                                           const double *__restrict__ tw,
                                                           const uint8_t *__restrict__ dang, double *x, double *y,
                                                           double *mass, int *iters, int *remaining) {
    cg::grid_group grid = cg::this_grid();
    __shared__ double sh[kCompT / 32];
    constexpr int RPW = 32 / VEC, NW = kCompT / 32;
    const int lane = threadIdx.x & 31, sub = lane / VEC, lv = lane % VEC, warp = threadIdx.x >> 5;
    for (int32_t c = blockIdx.x; c < n_comp; c += gridDim.x) {
        const int64_t lo = comp[2 * c], hi = comp[2 * c + 1];
        const double x0 = 1.0 / (double)(hi - lo);
        double dl = 0.0;
        for (int64_t i = lo + threadIdx.x; i < hi; i += kCompT) {
            x[i] = x0;
            if (dang[i]) dl += x0;
        }
        const double D = comp_block_sum(dl, sh);
        if (threadIdx.x == 0) {
            mass[c] = D;
            iters[c] = 0;
        }
    }
    grid.sync();
    // the warp's run of row groups and the component it starts in
    const int64_t total = goff[n_comp], nw = (int64_t)gridDim.x * NW, gw = (int64_t)blockIdx.x * NW + warp;
    const int64_t g0 = total * gw / nw, g1 = total * (gw + 1) / nw;
    int32_t c0 = 0, ch = n_comp - 1;
    while (c0 < ch) {
        const int32_t mid = c0 + ((ch - c0 + 1) >> 1);
        if (goff[mid] <= g0)
            c0 = mid;
        else
            ch = mid - 1;
    }
    for (int iter = 1;; iter++) {
        // iters[c]: minus the iterations run while the component goes on, their number once it has stopped
        int32_t c = c0;
        for (int64_t g = g0; g < g1;) {
            while (goff[c + 1] <= g) c++;
            const int64_t stop = min(g1, goff[c + 1]);
            if (__ldcg(iters + c) > 0) {
                g = stop;
                continue;
            }
            const int64_t hi = comp[2 * c + 1], base = comp[2 * c];
            const double coef = kAlpha + kBeta * __ldcg(mass + c);
            for (; g < stop; g++) {
                const int64_t r = base + (g - goff[c]) * RPW + sub;
                double acc = 0.0;
                if (r < hi) {
                    const int64_t e = in_off[r + 1];
                    for (int64_t k = in_off[r] + lv; k < e; k += VEC) acc += kBeta * in_w[k] * x[in_src[k]];
                }
#pragma unroll
                for (int o = VEC / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
                if (r < hi && lv == 0) y[r] = coef * tw[r] + acc;
            }
        }
        grid.sync();
        for (c = blockIdx.x; c < n_comp; c += gridDim.x) {
            if (__ldcg(iters + c) > 0) continue;  // uniform over the block
            const int64_t lo = comp[2 * c], hi = comp[2 * c + 1];
            double ls = 0.0;
            if (lv == 0) {
#pragma unroll 8
                for (int64_t r = lo + (int64_t)warp * RPW + sub; r < hi; r += (int64_t)NW * RPW) ls += __ldcg(y + r);
            }
            const double S = comp_block_sum(ls, sh);
            double el = 0.0, dl = 0.0;
#pragma unroll 4
            for (int64_t i = lo + threadIdx.x; i < hi; i += kCompT) {
                const double xn = __ldcg(y + i) / S;
                el += fabs(xn - x[i]);
                x[i] = xn;
                if (dang[i]) dl += xn;
            }
            const double diff = comp_block_sum(el, sh);
            const double D = comp_block_sum(dl, sh);
            if (threadIdx.x == 0) {
                const bool done = iter >= 200 || (diff <= 1.0e-15 && iter >= 50);  // Module.cpp:460
                mass[c] = D;
                iters[c] = done ? iter : -iter;
                if (!done) atomicAdd(remaining + iter, 1);
            }
        }
        grid.sync();
        if (__ldcg(remaining + iter) == 0) break;  // the same in every block
    }
}

// Copies of a graph share its flow: p of every non-canonical instance is read
// from its canonical copy.
__global__ void k_replicate_flows(int32_t n, const int32_t *node_inst, const int64_t *inst_noff,
                                  const int32_t *inst_canon, double *p) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t k = node_inst[i], c = inst_canon[k];
        if (c != k) p[i] = p[i - inst_noff[k] + inst_noff[c]];
    }
}

template <int VEC>
static void launch_power_union(int32_t n_comp, const int64_t *comp, const int64_t *goff, const int64_t *in_off,
                               const int32_t *in_src, const double *in_w, const double *tw, const uint8_t *dangling,
                               double *p, double *y, double *mass, int *iters, int *remaining, cudaStream_t s) {
    int per_sm = 0;
    RMX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_power_union<VEC>, kCompT, 0));
    if (per_sm < 1) throw CudaError(cudaErrorLaunchOutOfResources, "power iteration does not fit an SM");
    void *args[] = {(void *)&n_comp, (void *)&comp, (void *)&goff, (void *)&in_off, (void *)&in_src,
                    (void *)&in_w,   (void *)&tw,   (void *)&dangling, (void *)&p,  (void *)&y,
                    (void *)&mass,   (void *)&iters, (void *)&remaining};
    RMX_CUDA(cudaLaunchCooperativeKernel((void *)k_power_union<VEC>, dim3(std::min(per_sm, 4) * num_sms()),
                                         dim3(kCompT), args, 0, s));
    RMX_LAUNCHED();
}

int power_iteration_components(int32_t n, int32_t n_comp, const int64_t *comp, const int64_t *comp_dev,
                               const int32_t *node_inst, const int64_t *inst_noff, const int32_t *inst_canon,
                               const int64_t *in_off, const int32_t *in_src, const double *in_w, const double *tw,
                               const uint8_t *dangling, double *p, Arena &ar, cudaStream_t s, int vec) {
    if (n <= 0 || n_comp <= 0) return 0;
    size_t mk = ar.mark();
    double *y = ar.alloc<double>(n), *mass = ar.alloc<double>(n_comp);
    int *iters = ar.alloc<int>(n_comp), *remaining = ar.alloc<int>(256);
    const int rpw = 32 / vec;
    std::vector<int64_t> goff(n_comp + 1, 0);
    for (int32_t c = 0; c < n_comp; c++) goff[c + 1] = goff[c] + (comp[2 * c + 1] - comp[2 * c] + rpw - 1) / rpw;
    int64_t *d_goff = ar.alloc<int64_t>(n_comp + 1);
    RMX_CUDA(cudaMemcpyAsync(d_goff, goff.data(), sizeof(int64_t) * (n_comp + 1), cudaMemcpyHostToDevice, s));
    RMX_CUDA(cudaMemsetAsync(remaining, 0, sizeof(int) * 256, s));
    switch (vec) {
        case 4: launch_power_union<4>(n_comp, comp_dev, d_goff, in_off, in_src, in_w, tw, dangling, p, y, mass, iters, remaining, s); break;
        case 8: launch_power_union<8>(n_comp, comp_dev, d_goff, in_off, in_src, in_w, tw, dangling, p, y, mass, iters, remaining, s); break;
        case 16: launch_power_union<16>(n_comp, comp_dev, d_goff, in_off, in_src, in_w, tw, dangling, p, y, mass, iters, remaining, s); break;
        default: launch_power_union<32>(n_comp, comp_dev, d_goff, in_off, in_src, in_w, tw, dangling, p, y, mass, iters, remaining, s); break;
    }
    k_replicate_flows<<<blocks_for(n, 256, num_sms() * 32), 256, 0, s>>>(n, node_inst, inst_noff, inst_canon, p);
    RMX_LAUNCHED();
    std::vector<int> h(n_comp);
    RMX_CUDA(cudaMemcpyAsync(h.data(), iters, sizeof(int) * n_comp, cudaMemcpyDeviceToHost, s));
    RMX_CUDA(cudaStreamSynchronize(s));
    ar.release(mk);
    return *std::max_element(h.begin(), h.end());
}

// About 2.5 links per lane: more rows in flight per warp hide the gather
// latency better than idle lanes do (mean in-degree 20: 8 lanes, 6.7 ms
// against 9.2 ms with 16 lanes for 50 iterations on 19.5M links; R-MAT scale
// 24, mean 15.7: 4 lanes 7% faster than 8, 16 lanes 10% slower).
int spmv_width(double mean_in_degree) {
    return mean_in_degree <= 16 ? 4 : (mean_in_degree <= 24 ? 8 : (mean_in_degree <= 48 ? 16 : 32));
}

int power_iteration(int32_t n, int64_t m, const int64_t *in_off, const int32_t *in_src, const double *in_w, const double *tw,
                    const uint8_t *dangling, double *p, Arena &ar, cudaStream_t s, int vec, double alpha) {
    if (n <= 0) return 0;
    switch (vec) {
        case 4: return launch_power<4>(n, m, in_off, in_src, in_w, tw, dangling, p, ar, s, alpha);
        case 8: return launch_power<8>(n, m, in_off, in_src, in_w, tw, dangling, p, ar, s, alpha);
        case 16: return launch_power<16>(n, m, in_off, in_src, in_w, tw, dangling, p, ar, s, alpha);
        default: return launch_power<32>(n, m, in_off, in_src, in_w, tw, dangling, p, ar, s, alpha);
    }
}

// ------------------------------------------------------------ flows

// Edge flows f = p_u * w~ (Module.cpp:275-286) in FP64 and fixed point, and
// each node's unit statistics; the out-flow sum is a fixed-point (exact,
// order-free) sum, so heavy rows done by the whole warp give the same bits.
__global__ void k_flow_rows(int32_t n, const int64_t *off, double *f, fx_t *fx, const double *p, const double *tw,
                            const uint8_t *dangling, Stat4 *attr, fx_t *s0) {
    const int lane = threadIdx.x & 31;
    const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    fx_t s0l = 0;
    for (int64_t base = gw * 32; base < n; base += nw * 32) {
        const int64_t i = base + lane;
        bool heavy = false;
        fx_t out = 0;
        if (i < n) {
            const int64_t b = off[i], e = off[i + 1];
            heavy = e - b > kRowSeqMax;
            const double pi = p[i];
            if (!heavy)
                for (int64_t j = b; j < e; j++) {
                    const double v = pi * f[j];  // Module.cpp:280
                    f[j] = v;
                    const fx_t q = to_fx(v);
                    fx[j] = q;
                    out += q;
                }
            s0l += to_fxl(plogp(pi));
        }
        for (unsigned hv = __ballot_sync(kFull, heavy); hv; hv &= hv - 1) {
            const int src = __ffs(hv) - 1;
            const int64_t r = base + src;
            const int64_t b = off[r], e = off[r + 1];
            const double pr = p[r];
            fx_t o = 0;
            for (int64_t j = b + lane; j < e; j += 32) {
                const double v = pr * f[j];
                f[j] = v;
                const fx_t q = to_fx(v);
                fx[j] = q;
                o += q;
            }
#pragma unroll
            for (int q = 16; q > 0; q >>= 1) o += __shfl_xor_sync(kFull, o, q);
            if (lane == src) out = o;
        }
        if (i < n) {
            Stat4 a;
            a.P = to_fx(p[i]);
            a.TW = to_fx(tw[i]);
            a.D = dangling[i] ? a.P : 0;
            a.OUT = out;
            attr[i] = a;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s0l += __shfl_xor_sync(kFull, s0l, o);
    if (lane == 0 && s0l != 0) atomic_add_fx(s0, s0l);
}

__global__ void k_flow_cols(int64_t m, const int32_t *in_src, const double *in_w, const double *p, fx_t *in_fx) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x)
        in_fx[k] = to_fx(p[in_src[k]] * in_w[k]);
}

void edge_flows(int32_t n, int64_t m, const int64_t *out_off, double *out_f, fx_t *out_fx, const int32_t *in_src,
                const double *in_w, fx_t *in_fx, const double *p, const double *tw, const uint8_t *dangling,
                Stat4 *attr, fx_t *s0_acc, cudaStream_t s) {
    RMX_CUDA(cudaMemsetAsync(s0_acc, 0, sizeof(fx_t), s));
    k_flow_rows<<<blocks_for(n, 256, num_sms() * 32), 256, 0, s>>>(n, out_off, out_f, out_fx, p, tw, dangling, attr,
                                                                   s0_acc);
    RMX_LAUNCHED();
    if (m > 0) {
        k_flow_cols<<<blocks_for(m, 256, num_sms() * 32), 256, 0, s>>>(m, in_src, in_w, p, in_fx);
        RMX_LAUNCHED();
    }
}

// Singleton exit as Module::Module(int, Node*) (Module.cpp:76-95): the
// out-flow summed in link order, by the warp for heavy rows.
__global__ void k_singleton_exit(int32_t n, const int64_t *off, const double *f, const double *p, const double *tw,
                                 const uint8_t *dangling, double *ex) {
    const int lane = threadIdx.x & 31;
    const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t base = gw * 32; base < n; base += nw * 32) {
        const int64_t i = base + lane;
        bool heavy = false;
        double s = 0.0;
        if (i < n) {
            const int64_t b = off[i], e = off[i + 1];
            heavy = e - b > kRowSeqMax;
            if (!heavy)
                for (int64_t j = b; j < e; j++) s += f[j];
        }
        for (unsigned hv = __ballot_sync(kFull, heavy); hv; hv &= hv - 1) {
            const int src = __ffs(hv) - 1;
            const int64_t r = base + src;
            double t = 0.0;
            for (int64_t j = off[r] + lane; j < off[r + 1]; j += 32) t += f[j];
            t = warp_sum(t);
            if (lane == src) s = t;
        }
        if (i < n) ex[i] = dangling[i] ? (1.0 - tw[i]) * p[i] : kAlpha * (1.0 - tw[i]) * p[i] + kBeta * s;
    }
}

void singleton_exits(int32_t n, const int64_t *out_off, const double *out_f, const double *p, const double *tw,
                     const uint8_t *dangling, double *exitpr, cudaStream_t s) {
    k_singleton_exit<<<blocks_for(n, 256, num_sms() * 32), 256, 0, s>>>(n, out_off, out_f, p, tw, dangling, exitpr);
    RMX_LAUNCHED();
}

}  // namespace rmx

// K_reg^{-1} v for every subdomain (Cluster.cpp:967-1040, 1648-1678: the
// local solves of the start and of the displacements), one right-hand side.
//
// v_d <- L_d^{-T} L_d^{-1} v_d with the factor panels of device.cuh.
//
// A cluster of C CTAs of 8 warps works on one subdomain as a dataflow over
// its 32-row blocks (the panels' blocks: interior blocks from row 0, b-set
// blocks from row nr).  One warp owns a block: it takes the 32 x 32 tiles of
// its block row (forward) or block column (backward) in the order in which
// their operands become known, substitutes with the diagonal block and sends its 32 results to every CTA of the cluster (st.async into their
// shared memory, completing a transaction barrier per block).  A tile is
// loaded before the wait for its operand, so the chain from block to block
// is a barrier, a 32-term product, the substitution and a shared-memory hop,
// and everything off the chain is a stream of the factor.  (Multiplying by
// the inverse of the diagonal block instead is shorter but not backward
// stable: K_reg is singular up to its six fix DOFs, and the residual it
// leaves moved an E-contrast-100 solve by 4 iterations.)  All results stay in
// shared memory, x_b in the place of y_b: between the passes the cluster meets
// once, so that within a pass no warp waits for another to have read.
//
// Bound by the factor's bytes, read twice, or for few or small subdomains by
// the chain of N / 32 blocks (2 us per block and direction).  Against one
// CTA per subdomain with a block-wide barrier per 32 rows, forward and
// backward: 8 subdomains of 648 DOFs 1.18 -> 0.09 ms; 64 uneven ones of up to
// 5 577 57 -> 1.41 ms; 512 of 2 187 (10 GB of factor, read twice) 12.7 ->
// 4.5 ms = 4.6 TB/s.
//
// Both kernels here multiply by the rounded reciprocal of a pivot, 1.5 ulp a
// quotient where a division leaves 0.5; the displacements' distance from a
// 64-bit direct solve is the stopping rule's either way.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>
#include <vector>

#include "device.cuh"
#include "htfeti.h"
#include "mbar.cuh"

namespace htf {

constexpr int KS_WARPS = 8;

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ uint32_t cluster_ctas() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// first phase of a barrier whose arrivals come from any CTA of the cluster; false on time-out
__device__ __forceinline__ bool bar_wait_cluster(uint64_t *bar) {
    uint32_t done = 0;
    for (unsigned it = 0; it < TC_WAIT_LIMIT; ++it) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0, %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(TC_WAIT_HINT_NS)
            : "memory");
        if (done) return true;
    }
    return false;
}

// lane l's value to slot[l] of every CTA of the cluster, counted on their bar
__device__ __forceinline__ void send_block(double *slot, uint64_t *bar, int lane, double value, uint32_t ctas) {
    const uint32_t a = smem_u32(slot + lane), b = smem_u32(bar);
    for (uint32_t c = 0; c < ctas; ++c)
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(map_to_cta(a, c)),
                     "l"(__double_as_longlong(value)), "r"(map_to_cta(b, c))
                     : "memory");
}

// 32 partial sums per lane -> lane l holds the warp's sum of p[l]
__device__ __forceinline__ double warp_transpose_sum(double (&p)[32], int lane) {
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) {
        const bool upper = lane & s;
#pragma unroll
        for (int q = 0; q < s; ++q) {
            const double send = upper ? p[q] : p[q + s];
            const double keep = upper ? p[q + s] : p[q];
            p[q] = keep + __shfl_xor_sync(0xffffffffu, send, s);
        }
    }
    return p[0];
}

__global__ void __launch_bounds__(KS_WARPS * 32, 1) k_ksolve(const SubDev *__restrict__ subs,
                                                            const int *__restrict__ order,
                                                            const double *__restrict__ K, double *__restrict__ v,
                                                            int max_blocks, int *__restrict__ err) {
    extern __shared__ __align__(16) double ks_sm[];
    const uint32_t C = cluster_ctas(), rank = cluster_rank();
    const SubDev &sd = subs[order[blockIdx.x / C]];
    const int nI = (sd.nr + 31) / 32, nblk = nI + sd.nt, nr = sd.nr;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double *xs = ks_sm;                                              // [max_blocks][32] results
    double *D = xs + 32 * max_blocks + warp * (32 * 33);             // this warp's diagonal block
    uint64_t *fwd = reinterpret_cast<uint64_t *>(xs + 32 * max_blocks + KS_WARPS * 32 * 33);
    uint64_t *bwd = fwd + max_blocks;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
        mbar_init(&fwd[b], 1);
        mbar_init(&bwd[b], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncthreads();
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
        mbar_expect_tx(&fwd[b], 32 * sizeof(double));
        mbar_expect_tx(&bwd[b], 32 * sizeof(double));
    }
    cluster_sync_all();

    double *x = v + sd.nfull_off;
    auto start = [&](int b) { return b < nI ? 32 * b : nr + 32 * (b - nI); };
    auto width = [&](int b) { return b < nI ? min(32, nr - 32 * b) : 32; };
    // diagonal block b into D: L(c, j) at D[c * 33 + j], zero outside the block; returns
    // 1 / L(lane, lane)
    auto load_diag = [&](int b) {
        const int s = start(b), w = width(b);
        const double *col = K + kcol(sd, s) + s + lane;               // (s + lane, s + c) at col[c ld]
        const long long ld = kld(sd, s);
        __syncwarp();
        const double r = lane < w ? 1.0 / col[lane * ld] : 0.0;
#pragma unroll 8
        for (int c = 0; c < 32; ++c) {
            if (lane > c) D[lane * 33 + c] = (c < w && lane < w) ? col[c * ld] : 0.0;
        }
        __syncwarp();
        return r;
    };
    bool ok = true;
    // forward: y_b = L_bb^{-1} (v_b - sum_{k < b} L_bk y_k)
    const int first = int(rank) * KS_WARPS + warp, step = KS_WARPS * int(C);
    for (int b = first; b < nblk && ok; b += step) {
        const int r0 = start(b), wb = width(b);
        const double f = lane < wb ? x[r0 + lane] : 0.0;
        const double rd = load_diag(b);
        const int row = r0 + min(lane, wb - 1);
        double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0, lA[32], lB[32];
        auto load = [&](double (&l)[32], int k) {
            const int c0 = start(k), wk = width(k);
            const double *col = K + kcol(sd, c0) + row;
            const long long ld = kld(sd, c0);
#pragma unroll
            for (int j = 0; j < 32; ++j) l[j] = j < wk ? col[j * ld] : 0.0;
        };
        auto apply = [&](const double (&l)[32], int k) {
            ok = ok && warp_agree(bar_wait_cluster(&fwd[k]));
            const double2 *yk = reinterpret_cast<const double2 *>(xs + 32 * k);
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                const double2 u = yk[j / 2], w = yk[j / 2 + 1];
                a0 += l[j] * u.x;
                a1 += l[j + 1] * u.y;
                a2 += l[j + 2] * w.x;
                a3 += l[j + 3] * w.y;
            }
        };
        if (b > 0) load(lA, 0);
        for (int k = 0; k < b && ok; k += 2) {
            if (k + 1 < b) load(lB, k + 1);
            apply(lA, k);
            if (k + 1 < b) {
                if (k + 2 < b) load(lA, k + 2);
                apply(lB, k + 1);
            }
        }
        double y = lane < wb ? f - ((a0 + a1) + (a2 + a3)) : 0.0;
#pragma unroll
        for (int q = 0; q < 32; ++q) {
            if (lane == q) y *= rd;
            const double yq = __shfl_sync(0xffffffffu, y, q);
            if (lane > q) y -= D[lane * 33 + q] * yq;
        }
        if (ok) send_block(xs + 32 * b, &fwd[b], lane, y, C);
    }
    // x_b goes to the slots of y_b, and asynchronous stores have no order among themselves: no x is sent before
    // every y has landed in every CTA of the cluster (in a CTA that owns no later block nothing else waits for
    // y_b), by when no forward step reads one any more either
    for (int b = threadIdx.x; b < nblk && ok; b += blockDim.x) ok = bar_wait_cluster(&fwd[b]);
    ok = warp_agree(ok);
    cluster_sync_all();
    // backward: x_b = L_bb^{-T} (y_b - sum_{k > b} L_kb^T x_k)
    const int mine = first < nblk ? (nblk - 1 - first) / step : -1;
    for (int i = mine; i >= 0 && ok; --i) {
        const int b = first + i * step, c0 = start(b), wb = width(b);
        const double rd = load_diag(b);
        const double *col0 = K + kcol(sd, c0);
        const long long ld = kld(sd, c0);
        double z = xs[32 * b + lane], p[32], lA[32], lB[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) p[j] = 0.0;
        auto load = [&](double (&l)[32], int k) {
            const double *col = col0 + start(k) + min(lane, width(k) - 1);
#pragma unroll
            for (int j = 0; j < 32; ++j) l[j] = j < wb ? col[j * ld] : 0.0;
        };
        auto apply = [&](const double (&l)[32], int k) {
            // everything but the block just before is summed over the rows while that one is on its way
            if (k == b + 1) {
                z -= warp_transpose_sum(p, lane);
#pragma unroll
                for (int j = 0; j < 32; ++j) p[j] = 0.0;
            }
            ok = ok && warp_agree(bar_wait_cluster(&bwd[k]));
            const double xk = xs[32 * k + lane];                       // zero past the block's rows
#pragma unroll
            for (int j = 0; j < 32; ++j) p[j] += l[j] * xk;
        };
        if (b + 1 < nblk) load(lA, nblk - 1);
        for (int k = nblk - 1; k > b && ok; k -= 2) {
            if (k - 1 > b) load(lB, k - 1);
            apply(lA, k);
            if (k - 1 > b) {
                if (k - 2 > b) load(lA, k - 2);
                apply(lB, k - 1);
            }
        }
        z -= warp_transpose_sum(p, lane);
#pragma unroll
        for (int q = 31; q >= 0; --q) {
            if (lane == q) z *= rd;
            const double xq = __shfl_sync(0xffffffffu, z, q);
            if (lane < q) z -= D[q * 33 + lane] * xq;
        }
        if (!ok) break;
        send_block(xs + 32 * b, &bwd[b], lane, z, C);
        if (lane < wb) x[c0 + lane] = z;
    }
    // no CTA leaves while results are on their way to it
    if (warp == 0 && ok)
        for (int b = 0; b < nblk && ok; ++b) ok = warp_agree(bar_wait_cluster(&bwd[b]));
    if (!ok && lane == 0) atomicExch(err, HTF_ETIMEDOUT);
    cluster_sync_all();
}

__global__ void k_ksolve_multi(const SubDev *, const int *, const double *, double *, long long, int, const int *, int,
                               int *);

// shared memory of k_ksolve for subdomains of at most max_blocks 32-row blocks
size_t ksolve_smem(int max_blocks) {
    return (32 * size_t(max_blocks) + KS_WARPS * 32 * 33) * sizeof(double) + 2 * size_t(max_blocks) * sizeof(uint64_t);
}

// allows the kernel `optin` bytes (the device's limit, so that contexts of different sizes set the same value)
cudaError_t ksolve_prepare(int optin) {
    const cudaError_t e = cudaFuncSetAttribute(k_ksolve, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_ksolve_multi, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - 48 * 1024);
}

// CTAs per cluster for subdomains of blocks[i] 32-row blocks: the width with
// the shortest estimated time, one CTA per SM and no more CTAs than give
// every block of the largest subdomain a warp.  A subdomain takes the longer
// of its chain (KS_STEP_US per block and direction) and its factor, twice, at
// KS_CTA_GBS per CTA, and a third of the other; the launch the longest of its
// longest subdomain, the sum of CTA times over the SMs, and all factors at
// KS_GBS.  Measured: 8 subdomains of 21 blocks 118 us with one CTA each, 86
// with four; 64 uneven ones of up to 176 blocks 1.47 ms with four, 1.95 with
// eight; 512 of 71 blocks 4.5 ms with one.
int ksolve_ctas(const std::vector<int> &blocks) {
    constexpr double KS_STEP_US = 2.0, KS_CTA_GBS = 55.0, KS_GBS = 5000.0;
    const int most = blocks.empty() ? 1 : *std::max_element(blocks.begin(), blocks.end());
    int best = 1;
    double best_us = 0.0;
    for (int c = 1; c <= 8 && (c == 1 || KS_WARPS * (c / 2) < most); c *= 2) {
        double sum = 0.0, longest = 0.0, total = 0.0;
        for (int nb : blocks) {
            const double bytes = 8.0 * 32.0 * 32.0 * nb * (nb + 1.0);
            const double chain = 2.0 * KS_STEP_US * nb, stream = bytes / (c * KS_CTA_GBS * 1e3);
            const double us = std::max(chain, stream) + 0.3 * std::min(chain, stream);
            total += bytes;
            sum += c * us;
            longest = std::max(longest, us);
        }
        const double us = std::max(std::max(longest, sum / 148.0), total / (KS_GBS * 1e3));
        if (c == 1 || us < 0.98 * best_us) {
            best = c;
            best_us = us;
        }
    }
    return best;
}

// v_d <- K_reg,d^{-1} v_d for the nsub subdomains of `order` (largest first)
cudaError_t ksolve_launch(const SubDev *subs, const int *order, int nsub, const double *K, double *v, int max_blocks,
                          int ctas, int *err, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nsub * ctas);
    cfg.blockDim = dim3(KS_WARPS * 32);
    cfg.dynamicSmemBytes = ksolve_smem(max_blocks);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_ksolve, subs, order, K, v, max_blocks, err);
}

// ---------------------------------------------------------------------------
// Up to 32 right-hand sides per cluster (blockIdx.y: chunk of 32), the same
// dataflow with a CTA instead of a warp per 32-row block: X_b = L_bb^{-1}
// (V_b - sum_k L_bk X_k), then the transposed pass.  Results are exchanged
// through the vectors in global memory, with a barrier per block
// in every CTA of the cluster.  The 32 x 32 x 32 products run on the FP64
// tensor path out of double-buffered shared memory (both tiles column by
// column with a stride of 36 doubles: no bank conflicts), factor tiles
// prefetched two ahead into registers, X one ahead when it is known already;
// warp w owns row tiles 2 (w / 4), + 1 and one column tile, or, with up to
// 16 right-hand sides, a part of the k range of a column tile, the parts
// added in order.  (Fragments loaded straight from global memory touch eight
// lines per load and were bound by L1: 4.1 ms where this takes 2.2 for 64 x
// 2 187 DOFs and 32 right-hand sides; one CTA per subdomain took 7.4.)  Also
// the coarse problems' solves (plain N x N factors, clusters of one CTA, many
// chunks).
//
// Column j of subdomain d is at v + nfull_off + j * ld (ld = ldv, or N when
// ldv <= 0); nrhs columns, or ncols[d] when ncols is given.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void dmma_ks(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ bool bar_poll(uint64_t *bar) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_u32(bar))
        : "memory");
    return done;
}

// the CTA's global writes before the last __syncthreads are visible to whoever sees bar complete
__device__ __forceinline__ void publish(uint64_t *bar, uint32_t ctas) {
    __threadfence();
    for (uint32_t c = 0; c < ctas; ++c)
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(map_to_cta(smem_u32(bar), c))
                     : "memory");
}

__global__ void __launch_bounds__(256, 2) k_ksolve_multi(const SubDev *__restrict__ subs,
                                                         const int *__restrict__ order,
                                                         const double *__restrict__ K, double *v, long long ldv,
                                                         int nrhs, const int *__restrict__ ncols, int max_blocks,
                                                         int *__restrict__ err) {
    constexpr int S = 36;
    extern __shared__ __align__(16) uint64_t km_bars[];              // forward, then backward barriers
    __shared__ double Ls[32][33];                                    // diagonal block
    __shared__ __align__(16) double buf[4 * 32 * S];                 // two (factor, X) tile pairs; then the parts
    __shared__ double rinv[32];
    double(*T)[32][34] = reinterpret_cast<double(*)[32][34]>(buf);   // [4][32][34]: partial sums per k part
    const uint32_t C = cluster_ctas(), rank = cluster_rank();
    const int si = blockIdx.x / C;
    const SubDev &sd = subs[order ? order[si] : si];
    const bool plain = sd.K_bset < 0;
    const int nr = plain ? sd.N : sd.nr, nI = (nr + 31) / 32, nblk = nI + (plain ? 0 : sd.nt);
    const long long ld = ldv > 0 ? ldv : sd.N;
    const int col0 = 32 * blockIdx.y;
    const int nc = ncols ? min(32, ncols[si] - col0) : nrhs;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t4 = lane & 3;
    uint64_t *fwd = km_bars, *bwd = km_bars + max_blocks;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
        mbar_init(&fwd[b], 1);
        mbar_init(&bwd[b], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    cluster_sync_all();
    if (nc > 0) {
        double *x = v + sd.nfull_off + (size_t)col0 * ld;
        auto start = [&](int b) { return b < nI ? 32 * b : nr + 32 * (b - nI); };
        auto width = [&](int b) { return b < nI ? min(32, nr - 32 * b) : 32; };
        // column tiles in use and parts of the k range per column tile
        const int nct = nc <= 8 ? 1 : nc <= 16 ? 2 : 4, parts = 4 / nct;
        const int rt = 2 * (warp >> 2), ct = (warp & 3) % nct, part = (warp & 3) / nct;
        bool ok = true;
        double d[2][2];
        // sum over the tiles k = first, first + inc, .. (count of them) of A_k X_k; load_a(r, k, c): element (lane,
        // column c) of the factor tile; TR: A is its transpose.  Thread (lane, warp) stages columns warp, warp + 8, ..
        auto sweep = [&](auto tr, int first, int inc, int count, uint64_t *bars, auto &&load_a) {
            constexpr bool TR = decltype(tr)::value;
            double la[4], lb[4], xr[4];
            bool got = false;
            auto load_l = [&](double (&l)[4], int k) {
#pragma unroll
                for (int i = 0; i < 4; ++i) l[i] = load_a(k, warp + 8 * i);
            };
            auto load_x = [&](int k) {
                const int w = width(k), r0 = start(k);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int j = warp + 8 * i;
                    xr[i] = (lane < w && j < nc) ? __ldcg(x + r0 + lane + (size_t)j * ld) : 0.0;
                }
            };
            auto tile = [&](double (&l)[4], int i) {
                const int k = first + i * inc;
                double *At = buf + (i & 1) * (2 * 32 * S), *Xt = At + 32 * S;
                if (!got) {
                    if (ok) ok = bar_wait_cluster(&bars[k]);
                    load_x(k);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    At[(warp + 8 * q) * S + lane] = l[q];
                    Xt[(warp + 8 * q) * S + lane] = xr[q];
                }
                got = false;
                if (i + 1 < count && bar_poll(&bars[k + inc])) {
                    got = true;
                    load_x(k + inc);
                }
                if (i + 2 < count) load_l(l, k + 2 * inc);
                __syncthreads();
                auto mul = [&](int kg) {
                    const double b = Xt[(8 * ct + g) * S + 4 * kg + t4];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const double a = TR ? At[(8 * (rt + u) + g) * S + 4 * kg + t4]
                                            : At[(4 * kg + t4) * S + 8 * (rt + u) + g];
                        dmma_ks(d[u][0], d[u][1], a, b);
                    }
                };
                if (parts == 1) {
#pragma unroll
                    for (int kg = 0; kg < 8; ++kg) mul(kg);
                } else {
                    for (int kg = part * (8 / parts); kg < (part + 1) * (8 / parts); ++kg) mul(kg);
                }
            };
            d[0][0] = d[0][1] = d[1][0] = d[1][1] = 0.0;
            if (count > 0) load_l(la, first);
            if (count > 1) load_l(lb, first + inc);
            for (int i = 0; i < count; i += 2) {
                tile(la, i);
                if (i + 1 < count) tile(lb, i + 1);
            }
            __syncthreads();                                          // the tiles are consumed: buf takes the parts
        };
        auto load_diag = [&](int b) {
            const int s = start(b), w = width(b);
            const double *col = K + kcol(sd, s) + s + lane;
            const long long lk = kld(sd, s);
#pragma unroll
            for (int c = warp; c < 32; c += 8) Ls[lane][c] = (c <= lane && lane < w) ? col[c * lk] : 0.0;
            __syncthreads();
            if (threadIdx.x < 32) rinv[lane] = lane < w ? 1.0 / Ls[lane][lane] : 0.0;
        };
        // a[q]: row `lane`, column 4 warp + q of V_b (or Y_b) minus the product
        auto gather = [&](int r0, int w, double (&a)[4]) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                T[part][8 * (rt + u) + g][8 * ct + 2 * t4] = d[u][0];
                T[part][8 * (rt + u) + g][8 * ct + 2 * t4 + 1] = d[u][1];
            }
            __syncthreads();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int j = 4 * warp + q;
                double s = 0.0;
                if (j < 8 * nct) {
                    s = T[0][lane][j];
                    for (int p = 1; p < parts; ++p) s += T[p][lane][j];
                }
                a[q] = (lane < w && j < nc) ? __ldcg(x + r0 + lane + (size_t)j * ld) - s : 0.0;
            }
        };
        auto store = [&](int r0, int w, const double (&a)[4]) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int j = 4 * warp + q;
                if (lane < w && j < nc) x[r0 + lane + (size_t)j * ld] = a[q];
            }
            __syncthreads();
        };
        for (int b = int(rank); b < nblk; b += int(C)) {
            const int r0 = start(b), wb = width(b);
            load_diag(b);
            sweep(std::false_type(), 0, 1, b, fwd, [&](int k, int c) {
                const int s = start(k);
                return (c < width(k) && lane < wb) ? K[kcol(sd, s) + c * kld(sd, s) + r0 + lane] : 0.0;
            });
            double a[4];
            gather(r0, wb, a);
            if (4 * warp < nc)
                for (int p = 0; p < wb; ++p) {
                    const double rp = rinv[p], lp = Ls[lane][p];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const double y = __shfl_sync(0xffffffffu, a[q] * rp, p);
                        if (lane == p) a[q] = y;
                        else if (lane > p) a[q] -= lp * y;
                    }
                }
            store(r0, wb, a);
            if (threadIdx.x == 0) publish(&fwd[b], C);
        }
        // a result overwrites y_b only when every y is known, so when no forward step reads it any more
        for (int b = int(rank) + (nblk - 1 - int(rank)) / int(C) * int(C); b >= 0 && int(rank) < nblk; b -= int(C)) {
            const int r0 = start(b), wb = width(b);
            load_diag(b);
            if (ok) ok = bar_wait_cluster(&fwd[nblk - 1]);
            const double *colA = K + kcol(sd, r0) + lane;
            const long long lk = kld(sd, r0);
            sweep(std::true_type(), nblk - 1, -1, nblk - 1 - b, bwd, [&](int k, int c) {
                return (c < wb && lane < width(k)) ? colA[c * lk + start(k)] : 0.0;
            });
            double a[4];
            gather(r0, wb, a);
            if (4 * warp < nc)
                for (int p = wb - 1; p >= 0; --p) {
                    const double rp = rinv[p], lp = Ls[p][lane];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const double y = __shfl_sync(0xffffffffu, a[q] * rp, p);
                        if (lane == p) a[q] = y;
                        else if (lane < p) a[q] -= lp * y;
                    }
                }
            store(r0, wb, a);
            if (threadIdx.x == 0) publish(&bwd[b], C);
        }
        if (!ok && lane == 0) atomicExch(err, HTF_ETIMEDOUT);
    }
    cluster_sync_all();                                               // no CTA leaves while arrivals are on their way
}

// V <- K_reg^{-1} V (or the plain factors' inverse) for nsub matrices of at
// most max_blocks 32-row blocks and `chunks` chunks of 32 columns.  Clusters
// of up to 8 CTAs while all of them are resident (two per SM).
cudaError_t ksolve_multi_launch(const SubDev *subs, const int *order, int nsub, const double *K, double *v,
                                long long ldv, int nrhs, const int *ncols, int chunks, int max_blocks, int *err,
                                cudaStream_t s) {
    int ctas = 8;
    while (ctas > 1 && ((long long)nsub * chunks * ctas > 2 * 148 || ctas > max_blocks)) ctas /= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nsub * ctas, chunks);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = 2 * size_t(max_blocks) * sizeof(uint64_t);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_ksolve_multi, subs, order, K, v, ldv, nrhs, ncols, max_blocks, err);
}

}  // namespace htf

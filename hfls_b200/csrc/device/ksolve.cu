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
// shared memory, so no buffer is reused and no warp waits for another to
// have read.
//
// Bound by the factor's bytes, read twice, or for few or small subdomains by
// the chain of N / 32 blocks (2.7 us per block and direction).  Against one
// CTA per subdomain with a block-wide barrier per 32 rows, forward and
// backward: 8 subdomains of 648 DOFs 1.18 -> 0.12 ms; 64 uneven ones of up to
// 5 577 57 -> 1.46 ms; 512 of 2 187 (10 GB of factor, read twice) 12.7 ->
// 4.5 ms = 4.6 TB/s.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
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
            ok = ok && mbar_wait(&fwd[k], 0);
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
    // backward: x_b = L_bb^{-T} (y_b - sum_{k > b} L_kb^T x_k); a result x_k overwrites y_k's slot once
    // every y is known, when no forward step reads it any more
    const int mine = first < nblk ? (nblk - 1 - first) / step : -1;
    if (ok && mine >= 0) ok = mbar_wait(&fwd[nblk - 1], 0);
    for (int i = mine; i >= 0 && ok; --i) {
        const int b = first + i * step, c0 = start(b), wb = width(b);
        const double rd = load_diag(b);
        const double *col0 = K + kcol(sd, c0);
        const long long ld = kld(sd, c0);
        if (!mbar_wait(&fwd[b], 0)) { ok = false; break; }
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
            ok = ok && mbar_wait(&bwd[k], 0);
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
        for (int b = 0; b < nblk && ok; ++b) ok = mbar_wait(&bwd[b], 0);
    if (!ok && lane == 0) atomicExch(err, HTF_ETIMEDOUT);
    cluster_sync_all();
}

// shared memory of k_ksolve for subdomains of at most max_blocks 32-row blocks
size_t ksolve_smem(int max_blocks) {
    return (32 * size_t(max_blocks) + KS_WARPS * 32 * 33) * sizeof(double) + 2 * size_t(max_blocks) * sizeof(uint64_t);
}

// allows the kernel `optin` bytes (the device's limit, so that contexts of different sizes set the same value)
cudaError_t ksolve_prepare(int optin) {
    return cudaFuncSetAttribute(k_ksolve, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
}

// CTAs per cluster for subdomains of blocks[i] 32-row blocks: the width with
// the shortest estimated time, one CTA per SM.  A subdomain takes the longer
// of its chain (KS_STEP_US per block and direction) and its factor at
// KS_CTA_GBS per CTA and twice; the launch the longer of its longest
// subdomain and the sum of CTA times over the SMs.
int ksolve_ctas(const std::vector<int> &blocks) {
    constexpr double KS_STEP_US = 1.5, KS_CTA_GBS = 60.0;
    int best = 1;
    double best_us = 0.0;
    for (int c = 1; c <= 8; c *= 2) {
        double sum = 0.0, longest = 0.0;
        for (int nb : blocks) {
            const double bytes = 8.0 * 32.0 * 32.0 * nb * (nb + 1.0);
            const double us = std::max(2.0 * KS_STEP_US * nb, bytes / (c * KS_CTA_GBS * 1e3));
            sum += c * us;
            longest = std::max(longest, us);
        }
        const double us = std::max(longest, sum / 148.0);
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

}  // namespace htf

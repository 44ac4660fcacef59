// Setup kernels of the HTFETI path (FP64, sm_100a).
//
//  k_assemble        hex8 element stiffness (2x2x2 Gauss) and body-force
//                    load, scattered into the dense permuted K_d; elements of
//                    one colour share no node, so no atomics are needed.
//                    Restates Data::stf_mtrx_solid45 (Data.cpp:297-490) with
//                    the standard J^{-T} gradient and Data::feti_numeric
//                    (Data.cpp:231-273).
//  k_potrf_diag /    step-synchronous batched right-looking Cholesky: one
//  k_trsm_panel /    launch per 32-column step covers every subdomain that
//  k_syrk_update     still has that step (replaces the PARDISO factorisation
//                    of K_reg, Matrix.cpp:1115-1202).
//  k_snapshot        copies S_reg - D_fix (Dirichlet) or K_bb (lumped) of the
//                    trailing block into packed tiles (Matrix.cpp:1708-1871).
//  k_trtri_step      X = L_bb^{-1}, one launch per 32-row block.
//  k_lauum_tiles     F = X^T X = (K_reg^{-1})_bb into packed tiles.
//  k_build_V/Fc      V = [F Bc_b^T, -R_b] and Fc_d = Bc_b F Bc_b^T
//                    (Cluster.cpp:150-185).
#include <cuda_runtime.h>
#include <cstdint>

#include "device.cuh"
#include "htfeti.h"
#include "mbar.cuh"

namespace htf {

// ---------------------------------------------------------------------------
// assembly
// ---------------------------------------------------------------------------
__constant__ double c_gp[8][3];      // Gauss points (Data.cpp:363-386 order)

// Gauss points +-0.577350269189626 (the reference's literal, Data.cpp:344)
cudaError_t set_gauss_points(cudaStream_t s) {
    const double pt = 0.577350269189626;
    const double gr[8] = {-pt, -pt, -pt, -pt, pt, pt, pt, pt}, gs[8] = {-pt, -pt, pt, pt, -pt, -pt, pt, pt},
                 gt[8] = {-pt, pt, -pt, pt, -pt, pt, -pt, pt};
    double gp[8][3];
    for (int g = 0; g < 8; ++g) { gp[g][0] = gr[g]; gp[g][1] = gs[g]; gp[g][2] = gt[g]; }
    return cudaMemcpyToSymbolAsync(c_gp, gp, sizeof(gp), 0, cudaMemcpyHostToDevice, s);
}

__global__ void k_assemble(const int *__restrict__ elist, int count, const double *__restrict__ ecoord,
                           const int *__restrict__ esub, const int *__restrict__ eperm,
                           const double *__restrict__ subE, const double *__restrict__ subnu,
                           const SubDev *__restrict__ subs, double *__restrict__ Kbuf,
                           double *__restrict__ fbuf, double bfx, double bfy, double bfz) {
    __shared__ double G[8][8][3];    // dN_a/dx_k at Gauss point g
    __shared__ double Nw[8][8];      // N_a * detJ
    __shared__ double W[8];          // detJ
    __shared__ int P[24];
    __shared__ double X[8][3];
    const int e = elist[blockIdx.x];
    const int t = threadIdx.x;
    if (t < 24) {
        X[t / 3][t % 3] = ecoord[24 * (size_t)e + t];
        P[t] = eperm[24 * (size_t)e + t];
    }
    __syncthreads();
    if (t < 8) {
        const double r = c_gp[t][0], s = c_gp[t][1], q = c_gp[t][2];
        const double rn[8] = {-1, 1, 1, -1, -1, 1, 1, -1};
        const double sn[8] = {-1, -1, 1, 1, -1, -1, 1, 1};
        const double tn[8] = {-1, -1, -1, -1, 1, 1, 1, 1};
        double dNr[8], dNs[8], dNt[8], N[8];
        for (int a = 0; a < 8; ++a) {
            dNr[a] = 0.125 * rn[a] * (1. + sn[a] * s) * (1. + tn[a] * q);
            dNs[a] = 0.125 * sn[a] * (1. + rn[a] * r) * (1. + tn[a] * q);
            dNt[a] = 0.125 * tn[a] * (1. + rn[a] * r) * (1. + sn[a] * s);
            N[a] = 0.125 * (1. + rn[a] * r) * (1. + sn[a] * s) * (1. + tn[a] * q);
        }
        // M[i][j] = d x_i / d r_j
        double M[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
        for (int a = 0; a < 8; ++a)
            for (int i = 0; i < 3; ++i) {
                M[i][0] += dNr[a] * X[a][i];
                M[i][1] += dNs[a] * X[a][i];
                M[i][2] += dNt[a] * X[a][i];
            }
        const double det = M[0][0] * (M[1][1] * M[2][2] - M[1][2] * M[2][1]) -
                           M[0][1] * (M[1][0] * M[2][2] - M[1][2] * M[2][0]) +
                           M[0][2] * (M[1][0] * M[2][1] - M[1][1] * M[2][0]);
        const double id = 1.0 / det;
        // Mi = M^{-1}: Mi[j][i] = d r_j / d x_i
        double Mi[3][3];
        Mi[0][0] = (M[1][1] * M[2][2] - M[1][2] * M[2][1]) * id;
        Mi[0][1] = -(M[0][1] * M[2][2] - M[0][2] * M[2][1]) * id;
        Mi[0][2] = (M[0][1] * M[1][2] - M[0][2] * M[1][1]) * id;
        Mi[1][0] = -(M[1][0] * M[2][2] - M[1][2] * M[2][0]) * id;
        Mi[1][1] = (M[0][0] * M[2][2] - M[0][2] * M[2][0]) * id;
        Mi[1][2] = -(M[0][0] * M[1][2] - M[0][2] * M[1][0]) * id;
        Mi[2][0] = (M[1][0] * M[2][1] - M[1][1] * M[2][0]) * id;
        Mi[2][1] = -(M[0][0] * M[2][1] - M[0][1] * M[2][0]) * id;
        Mi[2][2] = (M[0][0] * M[1][1] - M[0][1] * M[1][0]) * id;
        for (int a = 0; a < 8; ++a) {
            for (int i = 0; i < 3; ++i)      // dN/dx_i = sum_j dN/dr_j * dr_j/dx_i
                G[t][a][i] = dNr[a] * Mi[0][i] + dNs[a] * Mi[1][i] + dNt[a] * Mi[2][i];
            Nw[t][a] = N[a] * det;
        }
        W[t] = det;
    }
    __syncthreads();
    const int d = esub[e];
    const SubDev sd = subs[d];
    const double E = subE[d], nu = subnu[d];
    const double lam = E * nu / ((1. + nu) * (1. - 2. * nu));
    const double mu = E / (2. * (1. + nu));
    for (int idx = t; idx < 576; idx += blockDim.x) {
        const int I = idx % 24, J = idx / 24;
        const int pI = P[I], pJ = P[J];
        if (pI < pJ) continue;                      // lower triangle in permuted order
        const int i = I >> 3, a = I & 7, j = J >> 3, b = J & 7;
        double v = 0.0;
        for (int g = 0; g < 8; ++g) {
            double s = lam * G[g][a][i] * G[g][b][j] + mu * G[g][a][j] * G[g][b][i];
            if (i == j) s += mu * (G[g][a][0] * G[g][b][0] + G[g][a][1] * G[g][b][1] + G[g][a][2] * G[g][b][2]);
            v += s * W[g];
        }
        Kbuf[kidx(sd, pI, pJ)] += v;
    }
    if (fbuf && t < 24) {             // no fbuf: a re-assembly of the factor alone
        const int i = t >> 3, a = t & 7;
        const double bf = (i == 0) ? bfx : (i == 1) ? bfy : bfz;
        double v = 0.0;
        for (int g = 0; g < 8; ++g) v += bf * Nw[g][a];
        fbuf[sd.nfull_off + P[t]] += v;
    }
}

// K_reg = K + D_fix: double the diagonal at the fix DOFs (Matrix.cpp:1029-1057)
// and put the identity on the padded rows.
__global__ void k_regularize(SubDev *subs, int nsub, double *Kbuf) {
    const int d = blockIdx.x;
    if (d >= nsub) return;
    SubDev &sd = subs[d];
    if (threadIdx.x < 6) {
        const int f = sd.fix[threadIdx.x];
        const long long a = kidx(sd, f, f);
        const double v = Kbuf[a];
        sd.fix_diag[threadIdx.x] = v;
        Kbuf[a] = 2.0 * v;
    }
    for (int r = sd.nr + sd.nb + threadIdx.x; r < sd.N; r += blockDim.x) Kbuf[kidx(sd, r, r)] = 1.0;
}

// ---------------------------------------------------------------------------
// batched Cholesky steps of up to CHOL_STEP = 64 columns (two 32-column factor
// panels): the diagonal block in one CTA, the panel below it one row per
// thread, the trailing update keeping one accumulator per 32-column panel and
// subtracting them in turn in registers, so each trailing tile is read and
// written once per 64 columns.  The sums are those of two successive
// 32-column right-looking steps (per panel: Cholesky of the diagonal block,
// row-wise substitution, block update subtracting a 32-term sum), in their
// order; quotients by the pivots come from div_by (device.cuh).
// ---------------------------------------------------------------------------
// Thread t holds row t's 32 columns of the current panel in registers and
// eliminates column by column: the pivot's square root and the finished
// column go through shared memory, every later column of the row is one
// independent FMA.  Per element that is the order of the row-wise
// substitution (columns ascending).  64 columns of 8 subdomains 88 -> 39 us
// against the form with the block in shared memory; bound by 64 dependent
// square roots and quotients.
__global__ void __launch_bounds__(CHOL_STEP) k_potrf_diag(const StepDesc *__restrict__ st,
                                                          const SubDev *__restrict__ subs,
                                                          double *__restrict__ Kbuf, int *__restrict__ status) {
    __shared__ double A[CHOL_STEP][CHOL_STEP + 1];
    __shared__ __align__(16) double col[2][CHOL_STEP];   // the finished column's entries, by row
    __shared__ double piv[2], rpiv[2];
    __shared__ int bad;
    const StepDesc s = st[blockIdx.x];
    const SubDev &sd = subs[s.d];
    const int k = s.k, nb = s.nb, t = threadIdx.x;
    if (t == 0) bad = 0;
    // column c of the step at P0 + c ld0, or P1 + (c - TILE) ld1; sixteen loads in flight
    double *P0 = Kbuf + kcol(sd, k) + k + t, *P1 = nb > TILE ? Kbuf + kcol(sd, k + TILE) + k + t : P0;
    const long long ld0 = kld(sd, k), ld1 = kld(sd, k + TILE);
#pragma unroll 16
    for (int c = 0; c < TILE; ++c) A[t][c] = (c < nb && t < nb && t >= c) ? P0[c * ld0] : 0.0;
#pragma unroll 16
    for (int c = 0; c < TILE; ++c) A[t][TILE + c] = (TILE + c < nb && t < nb && t >= TILE + c) ? P1[c * ld1] : 0.0;
    __syncthreads();
    // Cholesky of the 32-column panel at o with n columns: rows o .. o + n - 1, and the panel's rows below up to nb
    auto panel = [&](int o, int n) {
        double a[TILE];
#pragma unroll
        for (int c = 0; c < TILE; ++c) a[c] = (t >= o && c < n) ? A[t][o + c] : 0.0;
        const int r = t - o;                        // row within the panel
#pragma unroll
        for (int j = 0; j < TILE; ++j) {
            if (j < n) {                            // uniform
                if (r == j) {
                    double d = a[j];
                    if (!(d > 0.0)) {
                        if (!bad) bad = k + o + j + 1;
                        d = 1.0;
                    }
                    a[j] = sqrt(d);
                    piv[j & 1] = a[j];
                    rpiv[j & 1] = rsqrt(d);         // beside the square root, not after it: 1 / a[j] to 2 ulp
                }
                __syncthreads();
                if (r > j) a[j] = div_by(a[j], piv[j & 1], rpiv[j & 1]);
                if (r >= 0 && r < TILE) col[j & 1][r] = a[j];
                __syncthreads();
#pragma unroll
                for (int c = j + 1; c < TILE; ++c)
                    if (c <= r && c < n) a[c] -= a[j] * col[j & 1][c];
            }
        }
        __syncthreads();
        if (t >= o)
#pragma unroll
            for (int c = 0; c < TILE; ++c)
                if (c < n) A[t][o + c] = a[c];
        __syncthreads();
    };
    panel(0, min(nb, TILE));
    if (nb > TILE) {
        // block update of the second diagonal block, row TILE + lane, every other column per warp
        const int row = TILE + (t & 31);
        double x[TILE];
#pragma unroll
        for (int i = 0; i < TILE; ++i) x[i] = A[row][i];
        double upd[TILE / 2];
#pragma unroll
        for (int u = 0; u < TILE / 2; ++u) {
            const int c = TILE + 2 * u + (t >> 5);
            double acc = 0.0;
#pragma unroll
            for (int i = 0; i < TILE; ++i) acc += x[i] * A[c][i];
            upd[u] = acc;
        }
#pragma unroll
        for (int u = 0; u < TILE / 2; ++u) {
            const int c = TILE + 2 * u + (t >> 5);
            if (c <= row) A[row][c] -= upd[u];
        }
        __syncthreads();
        panel(TILE, nb - TILE);
    }
    if (t == 0 && bad) atomicCAS(&status[s.d], 0, bad);
#pragma unroll 8
    for (int c = 0; c < TILE; ++c) {
        if (t < nb && t >= c && c < nb) P0[c * ld0] = A[t][c];
        if (t < nb && t >= TILE + c) P1[c * ld1] = A[t][TILE + c];
    }
}

// rows below the diagonal block: x = x L_kk^{-T}, one row per thread, in
// registers, column by column: x_j is divided by the pivot and subtracted
// from the columns after it (independent FMAs; per element the columns
// ascend, as in the row-wise substitution), 32 columns at a time with one
// 32-term sum subtracted between the panels.  The factor's columns are
// broadcast from shared memory.  512 subdomains of 2 187 DOFs 29.6 -> 14.0 ms
// in all against dot products row by row with divisions; bound by the chain
// of quotients and by two CTAs per SM (registers).  grid: the step's row blocks of 128
// (flattened over its entries)
__global__ void __launch_bounds__(128) k_trsm_panel(const StepDesc *__restrict__ st, int cnt,
                                                    const SubDev *__restrict__ subs, double *__restrict__ Kbuf,
                                                    const int *__restrict__ hint) {
    __shared__ __align__(16) double L[CHOL_STEP][CHOL_STEP];         // [column][row]
    __shared__ double rinv[CHOL_STEP];
    const int e = step_entry(st, cnt, int(blockIdx.x), [](const StepDesc &x) { return x.rb0; }, hint);
    const StepDesc s = st[e];
    const int rb = int(blockIdx.x) - s.rb0;
    const SubDev &sd = subs[s.d];
    const int N = sd.N, k = s.k, nb = s.nb;
    const int row = k + nb + rb * blockDim.x + threadIdx.x;
    const bool in = row < N;
    const long long c0 = kcol(sd, k), c1 = nb > TILE ? kcol(sd, k + TILE) : c0;     // the step's two panels
    const long long ld0 = kld(sd, k), ld1 = kld(sd, k + TILE);
    {
        const int r = threadIdx.x % CHOL_STEP, h = threadIdx.x / CHOL_STEP;         // row, column parity
#pragma unroll
        for (int u = 0; u < CHOL_STEP / 2; ++u) {
            const int c = 2 * u + h;
            const double *P = Kbuf + (c < TILE ? c0 + c * ld0 : c1 + (c - TILE) * ld1) + k + r;
            L[c][r] = (r < nb && c < nb && c <= r) ? *P : 0.0;
        }
    }
    double x[CHOL_STEP];
#pragma unroll
    for (int j = 0; j < CHOL_STEP; ++j)
        x[j] = (in && j < nb) ? Kbuf[(j < TILE ? c0 + (long long)j * ld0 : c1 + (long long)(j - TILE) * ld1) + row] : 0.0;
    __syncthreads();
    if (threadIdx.x < CHOL_STEP) rinv[threadIdx.x] = int(threadIdx.x) < nb ? 1.0 / L[threadIdx.x][threadIdx.x] : 0.0;
    __syncthreads();
    if (!in) return;
#pragma unroll
    for (int j = 0; j < TILE; ++j)
        if (j < nb) {
            x[j] = div_by(x[j], L[j][j], rinv[j]);
#pragma unroll
            for (int c = j + 1; c < TILE; ++c) x[c] -= x[j] * L[j][c];
        }
    if (nb > TILE) {
        double acc[TILE];                           // block update by the first panel
#pragma unroll
        for (int c = 0; c < TILE; ++c) acc[c] = 0.0;
#pragma unroll
        for (int i = 0; i < TILE; ++i)
#pragma unroll
            for (int c = 0; c < TILE; ++c) acc[c] += x[i] * L[i][TILE + c];
#pragma unroll
        for (int c = 0; c < TILE; ++c) x[TILE + c] -= acc[c];
#pragma unroll
        for (int j = TILE; j < CHOL_STEP; ++j)
            if (j < nb) {
                x[j] = div_by(x[j], L[j][j], rinv[j]);
#pragma unroll
                for (int c = j + 1; c < CHOL_STEP; ++c) x[c] -= x[j] * L[j][c];
            }
    }
#pragma unroll
    for (int j = 0; j < CHOL_STEP; ++j)
        if (j < nb) Kbuf[(j < TILE ? c0 + (long long)j * ld0 : c1 + (long long)(j - TILE) * ld1) + row] = x[j];
}

// C (128 x 64 tile of the lower part of the trailing matrix) -= P_i P_j^T, P =
// the step's panel rows: 32 columns of P at a time, one sum per panel,
// subtracted in turn, C read and written once.  Steps come in pairs
// (StepDesc::pair): after the first only the second's columns are updated,
// after the second the rest with the panels of both.
//
// Persistent: one CTA per SM of eight product warps and four copy warps, which
// run through the step's tiles (CTA c takes tiles c, c + CTAs, ..).  The copy
// warps find the next tile and bring its panel rows (cp.async of 8 bytes: a
// column starts at any double) into one of two shared-memory stages while the
// product warps work on the other, C going straight to registers at the
// start of a tile and back from there; a tile's table look-ups, copies and C
// traffic thus hide behind the products of the tile before.  Products on the
// FP64 tensor path (mma.sync m8n8k4 .f64): warp w owns rows 32 (w / 2) .. +31
// and columns 32 (w % 2) .. +31, 4 x 4 tiles of 8 x 8, so a k-group of 4 is 8
// fragment loads for 16 MMAs; row strides of 132 and 68 doubles keep them
// free of bank conflicts.  C's loads are pinned to the start of the tile
// (left to the compiler they sink to their use: 128 ms).  One CTA per 64 x 64
// tile, with nothing in flight while it multiplied, reached 9.5 TFLOP/s on
// 512 x 2 187 DOFs (189 ms in all), this 19 (94 ms); 64 uneven subdomains of
// up to 5 577 DOFs 104 -> 50 ms.  The products alone would take 56 and 33 ms
// at the FP64 tensor rate (36 TFLOP/s); the rest is C through fragments of 64
// contiguous bytes.
__device__ __forceinline__ void dmma_syrk(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// 8-byte asynchronous copy global -> shared; src_bytes 0 writes a zero
__device__ __forceinline__ void cp_async8(double *dst, const double *src, int src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                     static_cast<unsigned>(__cvta_generic_to_shared(dst))),
                 "l"(src), "r"(src_bytes)
                 : "memory");
}

// *p, or zero: issued here, not where the value is used
__device__ __forceinline__ double ld_now(const double *p, bool in) {
    double v;
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %2, 0;\n\t"
        "mov.f64 %0, 0d0000000000000000;\n\t"
        "@q ld.global.f64 %0, [%1];\n\t}"
        : "=d"(v)
        : "l"(p), "r"(int(in)));
    return v;
}

constexpr int SYRK_LDA = 132, SYRK_LDB = 68;
constexpr int SYRK_STAGE = CHOL_STEP * (SYRK_LDA + SYRK_LDB);       // doubles: A columns, then B columns

struct SyrkTile {
    int d, k, nb;                           // subdomain (< 0: no more), panel columns of this stage
    int i0, j0, jend;                       // first row and column of the tile, end of the columns to update
    int part;                               // bit 0: the tile's first stage, bit 1: its last
};

__global__ void __launch_bounds__(SYRK_THREADS, 1) k_syrk_update(const StepDesc *__restrict__ st, int cnt, int tiles,
                                                                 const SubDev *__restrict__ subs, double *Kbuf,
                                                                 const int *__restrict__ hint, int *__restrict__ err) {
    extern __shared__ __align__(16) double syrk_sm[];                // two stages
    __shared__ __align__(8) uint64_t full[2], empty[2];
    __shared__ SyrkTile desc[2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int q = 0; q < 2; ++q) {
            mbar_init(&full[q], 32 * SYRK_COPY_WARPS + 1);     // the copy warps' lanes, the tile's description
            mbar_init(&empty[q], 8);
        }
    }
    __syncthreads();
    bool ok = true;
    // registers: 12 warps of 168 at launch, then 8 of 216 and 4 of 72 (the same sum)
    if (warp >= 8) {                        // copies: every SYRK_COPY_WARPS-th column
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        int n = 0, half = 0;
        StepDesc s{};
        for (int t = blockIdx.x; ok; t += half ? 0 : gridDim.x, ++n) {
            const int q = n & 1;
            SyrkTile T{-1, 0, 0, 0, 0, 0, 0};
            if (t < tiles) {
                if (half == 0) s = st[step_entry(st, cnt, t, [](const StepDesc &x) { return x.tri0; }, hint)];
                const int tri = t - s.tri0, t0 = s.k + s.nb;
                int bi = tri, bj = 0;                    // first of a pair: column block 0 of every row block
                if (s.pair <= 0) {
                    // row block bi (128 rows) has column blocks (64) 0 .. 2 bi + 1: bi (bi + 1) tiles before it
                    bi = (int)((sqrt(4.0 * tri + 1.0) - 1.0) * 0.5);
                    while ((bi + 1) * (bi + 2) <= tri) ++bi;
                    while (bi * (bi + 1) > tri) --bi;
                    bj = tri - bi * (bi + 1);
                }
                T = SyrkTile{s.d, s.k, s.nb, t0 + 128 * bi, t0 + 64 * bj, s.pair > 0 ? t0 + s.pair : subs[s.d].N, 3};
                if (s.pair < 0) {                        // the panels of both steps, one stage each
                    if (half == 0) {
                        T.k = s.k - CHOL_STEP;
                        T.nb = CHOL_STEP;
                    }
                    T.part = half == 0 ? 1 : 2;
                    half ^= 1;
                }
            }
            if (n >= 2) ok = warp_agree(mbar_wait(&empty[q], ((n >> 1) - 1) & 1));
            if (!ok) break;
            if (warp == 8 && lane == 0) desc[q] = T;
            if (T.d >= 0) {
                const SubDev &sd = subs[T.d];
                const int N = sd.N;
                double *A = syrk_sm + q * SYRK_STAGE, *B = A + CHOL_STEP * SYRK_LDA;
                for (int kc = 0; kc < T.nb; kc += TILE) {
                    // panel of columns k + kc ..: entry (row, k + kc + c) at P[row + c ld]
                    const double *P = Kbuf + kcol(sd, T.k + kc);
                    const long long ld = kld(sd, T.k + kc);
                    const int kn = min(TILE, T.nb - kc);
#pragma unroll 4
                    for (int c = warp - 8; c < TILE; c += SYRK_COPY_WARPS) {
                        const double *col = P + c * ld;
#pragma unroll
                        for (int r = 0; r < 128; r += 32) {
                            const bool in = c < kn && T.i0 + r + lane < N;
                            cp_async8(A + (kc + c) * SYRK_LDA + r + lane, in ? col + T.i0 + r + lane : Kbuf, in ? 8 : 0);
                        }
#pragma unroll
                        for (int r = 0; r < 64; r += 32) {
                            const bool in = c < kn && T.j0 + r + lane < N;
                            cp_async8(B + (kc + c) * SYRK_LDB + r + lane, in ? col + T.j0 + r + lane : Kbuf, in ? 8 : 0);
                        }
                    }
                }
            }
            if (warp == 8 && lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full[q])) : "memory");
            // each lane's arrival comes once its copies into this stage have landed
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full[q])) : "memory");
            if (T.d < 0) break;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
        const int g = lane >> 2, t4 = lane & 3;
        const int wr = 32 * (warp >> 1), wc = 32 * (warp & 1);
        // this thread's C: rows i0 + wr + 8 a + g, columns j0 + wc + 8 b + 2 t4 + h (lower part, in range)
        double *C[4][2];
        double c[4][4][2];
        int last[4][2];                     // rows row0 + 8 a of the column are stored for last <= row0 + 8 a < N
        int row0 = 0, N = 0;
        for (int n = 0;; ++n) {
            const int q = n & 1;
            ok = warp_agree(mbar_wait(&full[q], (n >> 1) & 1));
            if (!ok) break;
            const SyrkTile T = desc[q];
            if (T.d < 0) break;
            const double *A = syrk_sm + q * SYRK_STAGE, *B = A + CHOL_STEP * SYRK_LDA;
            if (T.part & 1) {
                const SubDev &sd = subs[T.d];
                N = sd.N;
                row0 = T.i0 + wr + g;
#pragma unroll
                for (int b = 0; b < 4; ++b)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int col = T.j0 + wc + 8 * b + 2 * t4 + h;
                        C[b][h] = Kbuf + kcol(sd, min(col, N - 1)) + row0;
                        last[b][h] = col < T.jend ? col : N;
#pragma unroll
                        for (int a = 0; a < 4; ++a)
                            c[a][b][h] = ld_now(C[b][h] + 8 * a, row0 + 8 * a >= last[b][h] && row0 + 8 * a < N);
                    }
            }
            for (int kc = 0; kc < T.nb; kc += TILE) {
                double acc[4][4][2];
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
                const int kgs = (min(TILE, T.nb - kc) + 3) >> 2;
#pragma unroll 2
                for (int kg = 0; kg < kgs; ++kg) {
                    const int kr = kc + 4 * kg + t4;
                    double av[4], bv[4];
#pragma unroll
                    for (int a = 0; a < 4; ++a) av[a] = A[kr * SYRK_LDA + wr + 8 * a + g];
#pragma unroll
                    for (int b = 0; b < 4; ++b) bv[b] = B[kr * SYRK_LDB + wc + 8 * b + g];
#pragma unroll
                    for (int a = 0; a < 4; ++a)
#pragma unroll
                        for (int b = 0; b < 4; ++b) dmma_syrk(acc[a][b][0], acc[a][b][1], av[a], bv[b]);
                }
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        c[a][b][0] -= acc[a][b][0];
                        c[a][b][1] -= acc[a][b][1];
                    }
            }
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&empty[q])) : "memory");
            if (!(T.part & 2)) continue;
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int a = 0; a < 4; ++a)
                        if (row0 + 8 * a >= last[b][h] && row0 + 8 * a < N) C[b][h][8 * a] = c[a][b][h];
        }
    }
    if (!ok && lane == 0) atomicExch(err, HTF_ETIMEDOUT);
}

// Copy the trailing nbp x nbp block into packed tiles, minus the fix diagonal.
__global__ void k_snapshot(const int *__restrict__ dlist, const SubDev *__restrict__ subs,
                           const double *__restrict__ Kbuf, double *__restrict__ Sbuf, long long t0) {
    const SubDev &sd = subs[dlist[blockIdx.x]];
    const int tile = blockIdx.y;
    if (tile >= sd.nt * (sd.nt + 1) / 2) return;
    int I = (int)((sqrt(8.0 * tile + 1.0) - 1.0) * 0.5);
    while ((I + 1) * (I + 2) / 2 <= tile) ++I;
    while (I * (I + 1) / 2 > tile) --I;
    const int J = tile - I * (I + 1) / 2;
    double *T = Sbuf + (sd.T_off - t0 + tile) * TILE_ELEMS;     // Sbuf holds the tiles from t0 on
    for (int idx = threadIdx.x; idx < TILE_ELEMS; idx += blockDim.x) {
        const int r = idx / TILE, c = idx % TILE;
        int gr = sd.nr + TILE * I + r, gc = sd.nr + TILE * J + c;
        if (gr < gc) { int tmp = gr; gr = gc; gc = tmp; }
        double v = Kbuf[kidx(sd, gr, gc)];
        if (gr == gc)
            for (int q = 0; q < 6; ++q)
                if (sd.fix[q] == gr) v -= sd.fix_diag[q];
        T[idx] = v;
    }
}

// acc(32 x 32) += A Xs on the FP64 tensor path (mma.sync m8n8k4): A = Ls
// (TR = false) or Ls^T (TR = true); warp w owns the 8-row tile w / 2 and the
// 8-column tiles 2 (w % 2), 2 (w % 2) + 1 (d[ct][h]: row 8 (w / 2) + lane / 4,
// column 8 (2 (w % 2) + ct) + 2 (lane % 4) + h).  Row stride 36 doubles: the
// fragment loads are conflict-free.
template <bool TR>
__device__ __forceinline__ void trsm_block_mma(const double (*Ls)[36], const double (*Xs)[36], int w, int lane,
                                               double (&d)[2][2]) {
    const int g = lane >> 2, t4 = lane & 3, rt = w >> 1, ct0 = 2 * (w & 1);
#pragma unroll
    for (int kg = 0; kg < 8; ++kg) {
        const int kr = 4 * kg + t4;
        const double a = TR ? Ls[kr][8 * rt + g] : Ls[8 * rt + g][kr];
#pragma unroll
        for (int ct = 0; ct < 2; ++ct) {
            const double b = Xs[kr][8 * (ct0 + ct) + g];
            asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                         : "+d"(d[ct][0]), "+d"(d[ct][1])
                         : "d"(a), "d"(b));
        }
    }
}

// ---------------------------------------------------------------------------
// X = L_bb^{-1}: block row i of X, all block columns j <= i
// ---------------------------------------------------------------------------
// (products out of double-buffered tiles, one barrier each, the next tile in
// registers; the substitution with one column per lane in registers: 23.0 ->
// 13.5 ms, 512 subdomains of 1 158 b rows)
__global__ void __launch_bounds__(256, 3) k_trtri_step(int i, const int *__restrict__ dlist,
                                                    const SubDev *__restrict__ subs,
                                                    const double *__restrict__ Kbuf, double *Xbuf) {
    constexpr int S = 36;
    __shared__ __align__(16) double At[2][32 * S];                   // L_i,kb and X_kb,j, column by column
    __shared__ __align__(16) double Xt[2][32 * S];
    __shared__ double rinv[32];
    const SubDev &sd = subs[dlist[blockIdx.x]];
    const int j = blockIdx.y;
    if (i >= sd.nt || j > i) return;
    const int nbp = sd.nbp, base = sd.nr;
    double *X = Xbuf + sd.X_off;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int g = lane >> 2, t4 = lane & 3, rt = w >> 1, ct0 = 2 * (w & 1);
    // sum_kb L_i,kb X_kb,j on the FP64 tensor path, then T = I - sum (block j = i) or -sum
    double d[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    double lr[4], xr[4], dr[4];
    auto fetch = [&](int kb) {
        const double *P = Kbuf + kcol(sd, base + 32 * kb) + base + 32 * i + lane;
        const long long ld = kld(sd, base + 32 * kb);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            lr[q] = P[(w + 8 * q) * ld];
            xr[q] = X[(32 * kb + lane) + (size_t)(32 * j + w + 8 * q) * nbp];
        }
    };
    {                                       // the diagonal block, needed at the end
        const double *P = Kbuf + kcol(sd, base + 32 * i) + base + 32 * i + lane;
        const long long ld = kld(sd, base + 32 * i);
#pragma unroll
        for (int q = 0; q < 4; ++q) dr[q] = w + 8 * q <= lane ? P[(w + 8 * q) * ld] : 0.0;
    }
    if (j < i) fetch(j);
    for (int kb = j; kb < i; ++kb) {
        double *A = At[(kb - j) & 1], *B = Xt[(kb - j) & 1];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            A[(w + 8 * q) * S + lane] = lr[q];
            B[(w + 8 * q) * S + lane] = xr[q];
        }
        __syncthreads();
        if (kb + 1 < i) fetch(kb + 1);
#pragma unroll
        for (int kg = 0; kg < 8; ++kg) {
            const double a = A[(4 * kg + t4) * S + 8 * rt + g];
#pragma unroll
            for (int ct = 0; ct < 2; ++ct)
                dmma_syrk(d[ct][0], d[ct][1], a, B[(8 * (ct0 + ct) + g) * S + 4 * kg + t4]);
        }
    }
    __syncthreads();
    double *La = At[0], *T = Xt[0];         // column by column again
#pragma unroll
    for (int q = 0; q < 4; ++q) La[(w + 8 * q) * S + lane] = dr[q];
#pragma unroll
    for (int ct = 0; ct < 2; ++ct)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = 8 * rt + g, c = 8 * (ct0 + ct) + 2 * t4 + h;
            T[c * S + r] = ((i == j && r == c) ? 1.0 : 0.0) - d[ct][h];
        }
    __syncthreads();
    if (tid < 32) rinv[tid] = 1.0 / La[tid * S + tid];
    __syncwarp();
    if (tid < 32) {                        // forward substitution, one column per lane
        double t[32];
#pragma unroll
        for (int r = 0; r < 32; ++r) t[r] = T[lane * S + r];
#pragma unroll
        for (int r = 0; r < 32; ++r) {
            t[r] = div_by(t[r], La[r * S + r], rinv[r]);
#pragma unroll
            for (int q = r + 1; q < 32; ++q) t[q] -= La[r * S + q] * t[r];
        }
#pragma unroll
        for (int r = 0; r < 32; ++r) T[lane * S + r] = t[r];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) X[(32 * i + lane) + (size_t)(32 * j + w + 8 * q) * nbp] = T[(w + 8 * q) * S + lane];
}

// F tile (I,J) = sum_{k >= I} X_kI^T X_kJ  (X lower triangular)
__global__ void __launch_bounds__(256) k_lauum_tiles(const int *__restrict__ dlist,
                                                     const SubDev *__restrict__ subs,
                                                     const double *__restrict__ Xbuf,
                                                     double *__restrict__ Fbuf) {
    __shared__ double A[32][36];
    __shared__ double B[32][36];
    const SubDev &sd = subs[dlist[blockIdx.x]];
    const int tile = blockIdx.y;
    if (tile >= sd.nt * (sd.nt + 1) / 2) return;
    int I = (int)((sqrt(8.0 * tile + 1.0) - 1.0) * 0.5);
    while ((I + 1) * (I + 2) / 2 <= tile) ++I;
    while (I * (I + 1) / 2 > tile) --I;
    const int J = tile - I * (I + 1) / 2;
    const double *X = Xbuf + sd.X_off;
    const int nbp = sd.nbp;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    // sum_kb X_kb,I^T X_kb,J on the FP64 tensor path (A = X_kb,I read transposed)
    double d[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    for (int kb = I; kb < sd.nt; ++kb) {
        for (int idx = tid; idx < 1024; idx += 256) {
            const int q = idx % 32, cc = idx / 32;
            A[q][cc] = X[(32 * kb + q) + (size_t)(32 * I + cc) * nbp];
            B[q][cc] = X[(32 * kb + q) + (size_t)(32 * J + cc) * nbp];
        }
        __syncthreads();
        trsm_block_mma<true>(A, B, w, lane, d);
        __syncthreads();
    }
    double *T = Fbuf + (sd.T_off + tile) * TILE_ELEMS;
    const int g = lane >> 2, t4 = lane & 3, rt = w >> 1, ct0 = 2 * (w & 1);
#pragma unroll
    for (int ct = 0; ct < 2; ++ct)
#pragma unroll
        for (int h = 0; h < 2; ++h) T[(8 * rt + g) * TILE + 8 * (ct0 + ct) + 2 * t4 + h] = d[ct][h];
}

// ---------------------------------------------------------------------------
// V = [F Bc_b^T, -R_b] and Fc_d = Bc_b V(:, 0:c)
// ---------------------------------------------------------------------------
__device__ __forceinline__ double tile_at(const double *F, const SubDev &sd, int i, int p) {
    int I = i / TILE, P = p / TILE;
    if (I >= P) return F[(sd.T_off + (long long)I * (I + 1) / 2 + P) * TILE_ELEMS + (i % TILE) * TILE + (p % TILE)];
    return F[(sd.T_off + (long long)P * (P + 1) / 2 + I) * TILE_ELEMS + (p % TILE) * TILE + (i % TILE)];
}

__global__ void k_build_V(const SubDev *__restrict__ subs, const double *__restrict__ Fbuf,
                          const int *__restrict__ bce_ptr, const int *__restrict__ bce_pos,
                          const double *__restrict__ bce_val, const double *__restrict__ Rbuf,
                          double *__restrict__ Vbuf) {
    const SubDev &sd = subs[blockIdx.x];
    const int col = blockIdx.y;
    if (col >= sd.c + 6) return;
    double *V = Vbuf + sd.V_off + (size_t)col * sd.nbp;
    if (col < sd.c) {
        const int e0 = bce_ptr[sd.bce_off + col], e1 = bce_ptr[sd.bce_off + col + 1];
        for (int i = threadIdx.x; i < sd.nbp; i += blockDim.x) {
            double v = 0.0;
            if (i < sd.nb)
                for (int e = e0; e < e1; ++e) v += bce_val[e] * tile_at(Fbuf, sd, i, bce_pos[e]);
            V[i] = v;
        }
    } else {
        const double *R = Rbuf + sd.R_off + (size_t)(col - sd.c) * sd.N;
        for (int i = threadIdx.x; i < sd.nbp; i += blockDim.x) V[i] = (i < sd.nb) ? -R[sd.nr + i] : 0.0;
    }
}

__global__ void k_build_Fc(const SubDev *__restrict__ subs, const double *__restrict__ Vbuf,
                           const int *__restrict__ bce_ptr, const int *__restrict__ bce_pos,
                           const double *__restrict__ bce_val, const long long *__restrict__ fc_off,
                           double *__restrict__ Fc) {
    const SubDev &sd = subs[blockIdx.x];
    const int c = sd.c;
    double *out = Fc + fc_off[blockIdx.x];
    for (int idx = threadIdx.x; idx < c * c; idx += blockDim.x) {
        const int r = idx % c, q = idx / c;
        const double *V = Vbuf + sd.V_off + (size_t)q * sd.nbp;
        double v = 0.0;
        for (int e = bce_ptr[sd.bce_off + r]; e < bce_ptr[sd.bce_off + r + 1]; ++e) v += bce_val[e] * V[bce_pos[e]];
        out[idx] = v;
    }
}

}  // namespace htf

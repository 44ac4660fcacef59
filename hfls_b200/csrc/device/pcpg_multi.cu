// Batched PCPG kernels: K load cases at once, vectors RHS-interleaved
// (entry (row, j) at row*K + j), one PcpgState per load case.  Each load
// case follows Cluster::pcpg (Cluster.cpp:1363-1458) independently; the
// matrices are read once per iteration for all K.  Reductions are
// fixed-order (deterministic).
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cstdint>

#include "device.cuh"

namespace htf {

// D += A B on the FP64 tensor path: one 8x8x4 product per warp.  Fragments:
// a = A[g][t4], b = B[t4][g], (d0, d1) = D[g][2 t4], D[g][2 t4 + 1] with
// g = lane / 4, t4 = lane % 4.
__device__ __forceinline__ void dmma_8x8x4(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// x_b = Bf^T w (optionally weighted; x_b itself only when xb != nullptr) for
// all K columns; also writes the X slabs of the tensor-core product: every
// column scaled by 2^EX_j (EX_j from the column's largest |w| times the bound
// xbound >= |x_b| / max|w|) as FP16 hi + lo, the hi plane (K rows x 64 B)
// then the lo plane, SWIZZLE_64B K-major.  One CTA per 32 consecutive slots
// (one K slab of one subdomain: b offsets and padded sizes are multiples of
// 32); the values go through shared memory so both outputs are written
// coalesced.  Two columns per thread and two slots per conversion (64
// subdomains of 8^3 elements, 32 columns, 1 964 CTAs, about 45 MB in L2): 17.1
// -> 13.6 us.
__global__ void __launch_bounds__(256) k_gather_multi(int nslots, int K, const int *__restrict__ ptr,
                                                      const int *__restrict__ ent, const double *w,
                                                      const double *__restrict__ weight, double *xb,
                                                      float *__restrict__ Xs, const unsigned *xmax, float xbound) {
    __shared__ double vs[32 * 33];
    __shared__ double sc[32];
    const int i0 = blockIdx.x * 32;
    pdl_next();
    const int K2 = K / 2, j2 = threadIdx.x % K2;    // a thread makes two columns of one or two slots
    int e0[2], e1[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int i = i0 + (int(threadIdx.x) + 256 * u) / K2;
        const bool here = 256 * u < 32 * K2 && i < nslots;
        e0[u] = here ? ptr[i] : 0;
        e1[u] = here ? ptr[i + 1] : 0;
    }
    pdl_wait();
    const double2 *w2 = reinterpret_cast<const double2 *>(w) + j2;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        if (256 * u >= 32 * K2) break;
        const int il = (int(threadIdx.x) + 256 * u) / K2, i = i0 + il;
        // a face slot has one entry, an edge slot three: their loads are in flight together
        int q[3];
        double2 v = make_double2(0.0, 0.0), a[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) q[k] = e0[u] + k < e1[u] ? ent[e0[u] + k] : -1;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            a[k] = q[k] >= 0 ? w2[(size_t)(q[k] >> 1) * K2] : make_double2(0.0, 0.0);
            if (weight && q[k] >= 0) {
                const double wt = weight[q[k] >> 1];
                a[k].x *= wt;
                a[k].y *= wt;
            }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (q[k] >= 0) {
                v.x += (q[k] & 1) ? -a[k].x : a[k].x;
                v.y += (q[k] & 1) ? -a[k].y : a[k].y;
            }
        for (int e = e0[u] + 3; e < e1[u]; ++e) {
            const int qe = ent[e], lam = qe >> 1;
            double2 ae = w2[(size_t)lam * K2];
            if (weight) {
                ae.x *= weight[lam];
                ae.y *= weight[lam];
            }
            v.x += (qe & 1) ? -ae.x : ae.x;
            v.y += (qe & 1) ? -ae.y : ae.y;
        }
        if (xb && i < nslots) reinterpret_cast<double2 *>(xb)[(size_t)i * K2 + j2] = v;
        vs[il * 33 + 2 * j2] = v.x;
        vs[il * 33 + 2 * j2 + 1] = v.y;
    }
    if (!Xs) return;
    // 2^EX_j, a normal FP64 number (EX_j comes from an FP32 value)
    if (threadIdx.x < K) sc[threadIdx.x] = __hiloint2double((1023 + tc_scale_exp(xmax[threadIdx.x], xbound)) << 20, 0);
    __syncthreads();
    // row j (load case) of each plane holds the 32 slots of this chunk, 64 bytes; a thread makes two slots of it
    __half2 *hi = reinterpret_cast<__half2 *>(Xs + (size_t)i0 * K);
    __half2 *lo = hi + 16 * K;
    for (int o = threadIdx.x; o < 16 * K; o += blockDim.x) {
        const int row = o / 16, c = 2 * (o % 16);
        const double v0 = vs[c * 33 + row] * sc[row], v1 = vs[(c + 1) * 33 + row] * sc[row];
        const __half h0 = __double2half(v0), h1 = __double2half(v1);
        const uint32_t b = uint32_t(row * 64 + c * 2);
        const uint32_t bs = (b ^ (((b >> 7) & 3u) << 4)) / 4;
        hi[bs] = __halves2half2(h0, h1);
        lo[bs] = __halves2half2(__double2half(v0 - (double)__half2float(h0)),
                                __double2half(v1 - (double)__half2float(h1)));
    }
}

// Partial V_d^T x_b over the 128-row chunk ch of subdomain d:
// tpart[(t_off + q) * nch + ch][j] = sum_{i in chunk} V_d[i][q] x_b[i][j]
// for q < c + 6 (QN >= c + 6 columns computed).  32-row pieces of V (stored
// q-major in shared memory) and x_b are staged, the next piece prefetched
// into registers; the products run on the FP64 tensor path, warp w owning
// the 8x8 output tiles w, w + 8, ... (q band = tile % (QN/8)).  Row strides
// of 36 and K + 4 doubles keep the fragment loads free of bank conflicts.
// CTA (subdomain, chunk), 256 threads.
template <int K, int QN>
__global__ void __launch_bounds__(256) k_vt_multi(int nch, const SubDev *__restrict__ subs,
                                                  const double *__restrict__ Vbuf, const double *xb,
                                                  double *tpart) {
    constexpr int VS = 36, XS = K + 4;
    constexpr int T = QN * K / 512;                 // 8x8 tiles per warp
    constexpr int UX = 32 * K / 256, UV = QN / 8;   // staged values per thread
    __shared__ double Vs[QN * VS];                  // [q][ii]
    __shared__ double Xs[32 * XS];                  // [ii][j]
    const SubDev &sd = subs[blockIdx.x];
    const int ch = blockIdx.y;
    const int ncol = sd.c + 6;
    const int r_end = min(sd.nb, ch * 128 + 128);
    const double *V = Vbuf + sd.V_off;
    const double *x = xb + (size_t)sd.xb_off * K;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int g = lane >> 2, t4 = lane & 3;
    double acc[T][2];
#pragma unroll
    for (int u = 0; u < T; ++u) acc[u][0] = acc[u][1] = 0.0;
    double xr[UX], vr[UV];
    auto fetch_x = [&](int i0) {
#pragma unroll
        for (int u = 0; u < UX; ++u) {
            const int o = threadIdx.x + 256 * u, ii = o / K;
            xr[u] = (i0 + ii < r_end) ? x[(size_t)(i0 + ii) * K + (o % K)] : 0.0;
        }
    };
    auto fetch_v = [&](int i0) {
#pragma unroll
        for (int u = 0; u < UV; ++u) {
            const int o = threadIdx.x + 256 * u, q = o / 32, ii = o % 32;
            vr[u] = (q < ncol && i0 + ii < r_end) ? V[(size_t)q * sd.nbp + i0 + ii] : 0.0;
        }
    };
    pdl_next();
    if (ch * 128 < r_end) fetch_v(ch * 128);
    pdl_wait();
    if (ch * 128 < r_end) fetch_x(ch * 128);
    for (int i0 = ch * 128; i0 < r_end; i0 += 32) {
#pragma unroll
        for (int u = 0; u < UX; ++u) {
            const int o = threadIdx.x + 256 * u;
            Xs[(o / K) * XS + o % K] = xr[u];
        }
#pragma unroll
        for (int u = 0; u < UV; ++u) {
            const int o = threadIdx.x + 256 * u;
            Vs[(o / 32) * VS + o % 32] = vr[u];
        }
        __syncthreads();
        if (i0 + 32 < r_end) {                      // next piece in flight during the products
            fetch_x(i0 + 32);
            fetch_v(i0 + 32);
        }
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
#pragma unroll
            for (int u = 0; u < T; ++u) {
                const int tile = warp + 8 * u, qb = tile % (QN / 8), jb = tile / (QN / 8);
                const double av = Vs[(8 * qb + g) * VS + 4 * kk + t4];
                const double bv = Xs[(4 * kk + t4) * XS + 8 * jb + g];
                dmma_8x8x4(acc[u][0], acc[u][1], av, bv);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < T; ++u) {
        const int tile = warp + 8 * u, qb = tile % (QN / 8), jb = tile / (QN / 8);
        const int q = 8 * qb + g, j = 8 * jb + 2 * t4;
        if (q < ncol) {
            double *o = tpart + (((size_t)sd.t_off + q) * nch + ch) * K + j;
            o[0] = acc[u][0];
            o[1] = acc[u][1];
        }
    }
}
#define HTF_VT(K, QN) \
    template __global__ void k_vt_multi<K, QN>(int, const SubDev *, const double *, const double *, double *);
HTF_VT(16, 32)
HTF_VT(16, 64)
HTF_VT(16, 128)
HTF_VT(32, 32)
HTF_VT(32, 64)
#undef HTF_VT

// gc[q][j] = sum over the t entries of coarse row q and their row chunks
__global__ void k_gc_multi(int ngc_total, int K, int nch, const int *__restrict__ gptr, const int *__restrict__ gidx,
                           const double *tpart, double *gc) {
    pdl_next();
    const long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const bool here = id < (long long)ngc_total * K;
    const int q = int(id / K), j = int(id % K);
    const int e0 = here ? gptr[q] : 0, e1 = here ? gptr[q + 1] : 0;
    int t = e0 < e1 ? gidx[e0] : 0;                 // the entry after this one is read ahead
    pdl_wait();
    if (!here) return;
    double s = 0.0;
    constexpr int U = 8;                            // chunks in flight
    for (int e = e0; e < e1; ++e) {
        const double *tp = tpart + (size_t)t * nch * K + j;
        if (e + 1 < e1) t = gidx[e + 1];
        for (int c0 = 0; c0 < nch; c0 += U) {
            double v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) v[u] = c0 + u < nch ? tp[(size_t)(c0 + u) * K] : 0.0;
#pragma unroll
            for (int u = 0; u < U; ++u) s += v[u];
        }
    }
    gc[(size_t)q * K + j] = s;
}

// S = M G per cluster (M symmetric ngc x ngc, G = gc ngc x K): CTA
// (cluster, 32-row block) of 128 threads; 32 x 64 tiles of M and 64-row
// tiles of G staged in shared memory, the next pair prefetched into
// registers.  Products on the FP64 tensor path: warp w owns rows
// 8w .. 8w + 7 and all K columns (K / 8 tiles sharing one A fragment).
template <int K>
__global__ void __launch_bounds__(128) k_coarse_multi(const ClusterDev *__restrict__ cl,
                                                      const double *__restrict__ Mbuf, const double *gc,
                                                      double *s) {
    constexpr int PK = 64, MS = PK + 4, GS = K + 4, NT = K / 8;
    constexpr int UM = 32 * PK / 128, UG = PK * K / 128;
    __shared__ double Ms[32 * MS];                  // [r][p]
    __shared__ double Gs[PK * GS];                  // [p][j]
    const ClusterDev c = cl[blockIdx.x];
    const int row0 = blockIdx.y * 32;
    if (row0 >= c.ngc) return;
    const double *M = Mbuf + c.M_off;
    const double *G = gc + (size_t)c.gc_off * K;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int g = lane >> 2, t4 = lane & 3;
    double acc[NT][2];
#pragma unroll
    for (int u = 0; u < NT; ++u) acc[u][0] = acc[u][1] = 0.0;
    double mr[UM], gr[UG];
    auto fetch_m = [&](int p0) {
#pragma unroll
        for (int u = 0; u < UM; ++u) {
            const int o = threadIdx.x + 128 * u, r = o / PK, pp = o % PK;
            mr[u] = (row0 + r < c.ngc && p0 + pp < c.ngc) ? M[(size_t)(row0 + r) * c.ngc + p0 + pp] : 0.0;
        }
    };
    auto fetch_g = [&](int p0) {
#pragma unroll
        for (int u = 0; u < UG; ++u) {
            const int o = threadIdx.x + 128 * u, pp = o / K;
            gr[u] = (p0 + pp < c.ngc) ? G[(size_t)(p0 + pp) * K + (o % K)] : 0.0;
        }
    };
    pdl_next();
    fetch_m(0);
    pdl_wait();
    fetch_g(0);
    for (int p0 = 0; p0 < c.ngc; p0 += PK) {
#pragma unroll
        for (int u = 0; u < UM; ++u) {
            const int o = threadIdx.x + 128 * u;
            Ms[(o / PK) * MS + o % PK] = mr[u];
        }
#pragma unroll
        for (int u = 0; u < UG; ++u) {
            const int o = threadIdx.x + 128 * u;
            Gs[(o / K) * GS + o % K] = gr[u];
        }
        __syncthreads();
        if (p0 + PK < c.ngc) {                      // next tiles in flight during the products
            fetch_m(p0 + PK);
            fetch_g(p0 + PK);
        }
#pragma unroll
        for (int kk = 0; kk < PK / 4; ++kk) {
            const double av = Ms[(8 * warp + g) * MS + 4 * kk + t4];
#pragma unroll
            for (int u = 0; u < NT; ++u)
                dmma_8x8x4(acc[u][0], acc[u][1], av, Gs[(4 * kk + t4) * GS + 8 * u + g]);
        }
        __syncthreads();
    }
    const int row = row0 + 8 * warp + g;
    if (row < c.ngc)
#pragma unroll
        for (int u = 0; u < NT; ++u) {
            double *o = s + ((size_t)c.gc_off + row) * K + 8 * u + 2 * t4;
            o[0] = acc[u][0];
            o[1] = acc[u][1];
        }
}
template __global__ void k_coarse_multi<16>(const ClusterDev *, const double *, const double *, double *);
template __global__ void k_coarse_multi<32>(const ClusterDev *, const double *, const double *, double *);

// The row kernels below (k_rows_multi, k_gf_apply_multi, the updates) run 128
// threads, thread (lr, j2) the columns 2 j2 and 2 j2 + 1 of the rows
// lr, lr + 256 / K, ...: 16-byte accesses, half the instructions per byte of
// one column per thread, by which these kernels (vectors in L2) are bound.  One
// column per thread -> two, alone: 64 subdomains of 8^3 elements, 32 columns:
// k_gf_apply_multi 14.7 -> 10.4 us, updates 11.0 -> 9.3 and 10.6 -> 8.3,
// k_rows_multi 10.1 -> 10.7; 32 uneven subdomains, 8 load cases in 16 columns:
// 6.3 -> 5.0, 5.5 -> 4.6, 5.3 -> 5.1, 5.2 -> 4.4 us.

// per-block, per-column tree sum of prod over the block's 256 / K rows -> partial[block][j]
__device__ __forceinline__ void block_col_partial(double2 prod, int K, double *partial) {
    __shared__ double2 red[128];
    const int K2 = K / 2, lr = threadIdx.x / K2, tid = threadIdx.x;
    red[tid] = prod;
    __syncthreads();
    for (int o = 128 / K; o > 0; o >>= 1) {
        if (lr < o) {
            red[tid].x += red[tid + o * K2].x;
            red[tid].y += red[tid + o * K2].y;
        }
        __syncthreads();
    }
    if (lr == 0) reinterpret_cast<double2 *>(partial)[(size_t)blockIdx.x * K2 + tid] = red[tid];
}

// out[r][j] = wt[r] * sum_k sign * y[slot][j]; partial dot with dotv per
// (block, j).  Blocks stride over groups of 256 / K rows (fixed assignment,
// so the partials and their sums are the same on every run); each thread
// has the loads of two of its rows in flight and adds them in row order.
__device__ __forceinline__ double2 row_value(int r, int K2, const int *__restrict__ rslot,
                                             const double *__restrict__ rsign, const double2 *yb,
                                             const double *__restrict__ weight) {
    const int2 sl = reinterpret_cast<const int2 *>(rslot)[r];
    const double2 sg = reinterpret_cast<const double2 *>(rsign)[r];
    const double wt = weight ? weight[r] : 1.0;
    const double2 zero = make_double2(0.0, 0.0);
    const double2 y0 = sl.x >= 0 ? yb[(size_t)sl.x * K2] : zero, y1 = sl.y >= 0 ? yb[(size_t)sl.y * K2] : zero;
    double2 v = zero;
    if (sl.x >= 0) {
        v.x += sg.x * y0.x;
        v.y += sg.x * y0.y;
    }
    if (sl.y >= 0) {
        v.x += sg.y * y1.x;
        v.y += sg.y * y1.y;
    }
    if (weight) {
        v.x *= wt;
        v.y *= wt;
    }
    return v;
}

// y_b -= V_d s_d for all K load cases of a batch vector: the coarse
// correction of the F apply (Cluster.cpp:1114-1188, y = F_d x_b - V_d s_d
// with V_d = [F_d Bc_d^T, -R_d], s_d the cluster coarse solution at the
// subdomain's Bc rows and alpha slot), after the tensor-core product so the
// product's CTAs end without an FP64 epilogue.  CTA (subdomain, 128-row
// chunk), a 128 x K by (c + 6) x K product: s_d staged in shared memory
// ((c + 6) K <= 2048 doubles, checked at set-up), V in chunks of 16 columns
// (coalesced column reads); thread (row group, case group) keeps 128 K / 256
// outputs in registers (rows rg + RG i, case pairs jg + JG c: conflict-free
// 16-byte shared-memory reads), summed over the columns in order.  y is read
// only for the subtraction, so that three CTAs fit an SM: the mixed iteration
// of 32 load cases 1744 -> 1688 us (512-subdomain cube), 271 -> 268 (64
// subdomains of 8^3 elements, this kernel 22 -> 20 us for 5 us of FP64
// operations).
template <int K>
__global__ void __launch_bounds__(256, 3) k_correct_multi(const SubDev *__restrict__ subs,
                                                       const ClusterDev *__restrict__ cl,
                                                       const double *__restrict__ V, const int *__restrict__ bcr,
                                                       const double *s, double *yb) {
    constexpr int QC = 16;                            // V columns per shared-memory chunk
    constexpr int JG = K / 4;                         // case groups (two pairs of cases per thread)
    constexpr int RG = 256 / JG;                      // row groups
    constexpr int RPT = 128 / RG;                     // rows per thread
    __shared__ double2 ss[1024];
    __shared__ double vs[QC][128];
    __shared__ int ps[2048 / K];
    const SubDev &sd = subs[blockIdx.x];
    const int r0 = blockIdx.y * 128;
    if (r0 >= sd.nb) return;
    const int nc = sd.c + 6;
    pdl_next();
    const int rend = min(128, sd.nb - r0);
    const int jg = threadIdx.x % JG, rg = threadIdx.x / JG;
    const double *Vd = V + sd.V_off + r0;
    double2 acc[RPT][2];
#pragma unroll
    for (int i = 0; i < RPT; ++i) acc[i][0] = acc[i][1] = make_double2(0.0, 0.0);
    // the next V chunk is loaded into registers while the current one multiplies
    constexpr int VPT = QC * 128 / 256;               // V values per thread and chunk
    double vr[VPT];
    auto fetch = [&](int q0) {
#pragma unroll
        for (int u = 0; u < VPT; ++u) {
            const int o = threadIdx.x + 256 * u, q = o >> 7, r = o & 127;
            vr[u] = (q0 + q < nc && r < rend) ? Vd[(size_t)(q0 + q) * sd.nbp + r] : 0.0;
        }
    };
    fetch(0);
    if (int(threadIdx.x) < nc)                        // (c + 6) K <= 2048
        ps[threadIdx.x] = cl[sd.cluster].gc_off + (int(threadIdx.x) < sd.c ? bcr[sd.bcr_off + threadIdx.x]
                                                                           : sd.alpha_pos + int(threadIdx.x) - sd.c);
    __syncthreads();
    pdl_wait();
    const double2 *s2 = reinterpret_cast<const double2 *>(s);
#pragma unroll 4
    for (int o = threadIdx.x; o < nc * (K / 2); o += 256) ss[o] = s2[(size_t)ps[o / (K / 2)] * (K / 2) + o % (K / 2)];
    double2 *y2 = reinterpret_cast<double2 *>(yb) + ((size_t)sd.xb_off + r0) * (K / 2) + jg;
    for (int q0 = 0; q0 < nc; q0 += QC) {
        const int qn = min(QC, nc - q0);
        __syncthreads();                              // s_d staged, the previous chunk consumed
#pragma unroll
        for (int u = 0; u < VPT; ++u) {
            const int o = threadIdx.x + 256 * u;
            vs[o >> 7][o & 127] = vr[u];
        }
        __syncthreads();
        if (q0 + QC < nc) fetch(q0 + QC);
#pragma unroll 2
        for (int q = 0; q < qn; ++q) {
            const double2 *sq = ss + (q0 + q) * (K / 2) + jg;
            const double2 s0 = sq[0], s1 = sq[JG];
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const double v = vs[q][rg + RG * i];
                acc[i][0].x += v * s0.x;
                acc[i][0].y += v * s0.y;
                acc[i][1].x += v * s1.x;
                acc[i][1].y += v * s1.y;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < RPT; ++i)
        if (rg + RG * i < rend)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                double2 &y = y2[(rg + RG * i) * (K / 2) + JG * c];
                y = make_double2(y.x - acc[i][c].x, y.y - acc[i][c].y);
            }
}

template __global__ void k_correct_multi<16>(const SubDev *, const ClusterDev *, const double *, const int *,
                                             const double *, double *);
template __global__ void k_correct_multi<32>(const SubDev *, const ClusterDev *, const double *, const int *,
                                             const double *, double *);

// dot2v (with dotv): also the partials of dot2v . dotv into partial2
__global__ void __launch_bounds__(128) k_rows_multi(int nlam, int K, const int *__restrict__ rslot,
                                                    const double *__restrict__ rsign, const double *yb,
                                                    const double *__restrict__ weight, double *out,
                                                    const double *dotv, double *partial, const double *dot2v,
                                                    double *partial2) {
    pdl_next();
    pdl_wait();
    const int rows_per_block = 256 / K, K2 = K / 2;
    const int lr = threadIdx.x / K2, j2 = threadIdx.x % K2;
    const int stride = gridDim.x * rows_per_block;
    const double2 *y2 = reinterpret_cast<const double2 *>(yb) + j2;
    const double2 *d2 = reinterpret_cast<const double2 *>(dotv) + j2;
    const double2 *g2 = reinterpret_cast<const double2 *>(dot2v) + j2;
    double2 *o2 = reinterpret_cast<double2 *>(out) + j2;
    const double2 zero = make_double2(0.0, 0.0);
    double2 prod = zero, prod2 = zero;
    for (int r0 = blockIdx.x * rows_per_block; r0 < nlam; r0 += 2 * stride) {
        double2 v[2], d[2], g[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int r = r0 + k * stride + lr;
            const bool here = r < nlam;
            v[k] = here ? row_value(r, K2, rslot, rsign, y2, weight) : zero;
            d[k] = here && dotv ? d2[(size_t)r * K2] : zero;
            g[k] = here && dot2v ? g2[(size_t)r * K2] : zero;
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int r = r0 + k * stride + lr;
            if (r >= nlam) continue;
            o2[(size_t)r * K2] = v[k];
            if (dotv) {
                prod.x += v[k].x * d[k].x;
                prod.y += v[k].y * d[k].y;
            }
            if (dot2v) {
                prod2.x += g[k].x * d[k].x;
                prod2.y += g[k].y * d[k].y;
            }
        }
    }
    if (partial) block_col_partial(prod, K, partial);
    if (dot2v) {
        __syncthreads();
        block_col_partial(prod2, K, partial2);
    }
}

// Gf^T x per chunk and column.  Of the 256 / K interleaved sums of a chunk
// (entries lr, lr + 256/K, ...) CTA (chunk, p) makes those with lr % 4 == p:
// its rows and Gf values (up to 256 entries) are staged in shared memory before
// the wait, thread (lr / 4, j) walks its entries with 32 x loads in flight, and
// the sums are added as a tree; k_gt_sum_multi adds the four parts the same
// way.  Bound by the latency of the x loads, a row of K values each: 60 chunks
// are 240 CTAs in four parts.  64 subdomains of 8^3 elements, 32 columns (60
// chunks), alone: 15.8 us with one CTA per chunk, 9.8 us in parts.
constexpr int GFT_PART = 1024 / 4;                 // most entries of a part of a chunk
__global__ void __launch_bounds__(64) k_gft_partial_multi(int K, const int *__restrict__ chunk_beg,
                                                          const int *__restrict__ chunk_end,
                                                          const int *__restrict__ crow,
                                                          const double *__restrict__ cval,
                                                          const double *x,
                                                          double *partial) {
    __shared__ double2 cs[3 * GFT_PART];            // then [6][64] sums
    __shared__ int rs[GFT_PART];
    const int ch = blockIdx.x / 4, p = blockIdx.x % 4, tid = threadIdx.x;
    const int j = tid % K, nl = 64 / K, lr = tid / K;
    const int beg = chunk_beg[ch] + p, n = (chunk_end[ch] - beg + 3) / 4;
    pdl_next();
    const double2 *cv = reinterpret_cast<const double2 *>(cval);
#pragma unroll
    for (int u = 0; u < GFT_PART / 64; ++u) {       // missing entries: zeros
        const int o = tid + 64 * u;
        rs[o] = o < n ? crow[beg + 4 * o] : -1;
    }
#pragma unroll
    for (int u = 0; u < 3 * GFT_PART / 64; ++u) {
        const int o = tid + 64 * u, e = o / 3;
        cs[o] = e < n ? cv[3 * (size_t)(beg + 4 * e) + o % 3] : make_double2(0.0, 0.0);
    }
    pdl_wait();
    __syncthreads();
    double s[6] = {0, 0, 0, 0, 0, 0};
    constexpr int U = 32;                           // of at most 128 (K = 32) or 64 entries per thread
    for (int e0 = lr; e0 < n; e0 += U * nl) {
        double xv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int r = rs[e0 + u * nl];
            xv[u] = r >= 0 ? x[(size_t)r * K + j] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const double2 *c = cs + 3 * (e0 + u * nl);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                s[2 * q] += c[q].x * xv[u];
                s[2 * q + 1] += c[q].y * xv[u];
            }
        }
    }
    __syncthreads();                                // the staged values are consumed
    double *red = reinterpret_cast<double *>(cs);
#pragma unroll
    for (int q = 0; q < 6; ++q) red[q * 64 + tid] = s[q];
    __syncthreads();
    for (int o = nl / 2; o > 0; o >>= 1) {
        if (lr < o)
#pragma unroll
            for (int q = 0; q < 6; ++q) red[q * 64 + tid] += red[q * 64 + tid + o * K];
        __syncthreads();
    }
    if (lr == 0)
#pragma unroll
        for (int q = 0; q < 6; ++q) partial[((size_t)blockIdx.x * 6 + q) * K + j] = red[q * 64 + j];
}

// gt[c][i][j] = sum of the chunk partials of cluster c (in chunk order); CTA
// (cluster, mode i): 32 chunks at a time are read by all threads (four parts
// each, as a tree) and added in order by thread j
__global__ void __launch_bounds__(256) k_gt_sum_multi(int K, const int *__restrict__ cl_chunk_ptr,
                                                      const double *gpart, double *gt) {
    __shared__ double v[32 * 32];
    pdl_next();
    const int c = blockIdx.x / 6, i = blockIdx.x % 6, j = threadIdx.x % K, lr = threadIdx.x / K, nl = 256 / K;
    const int beg = cl_chunk_ptr[c], end = cl_chunk_ptr[c + 1];
    pdl_wait();
    double s = 0.0;
    for (int c0 = beg; c0 < end; c0 += 32) {
        const int n = min(32, end - c0);
#pragma unroll 4
        for (int o = lr; o < n; o += nl) {
            const double *g = gpart + ((size_t)(c0 + o) * 24 + i) * K + j;
            v[o * K + j] = (g[0] + g[12 * K]) + (g[6 * K] + g[18 * K]);
        }
        __syncthreads();
        if (lr == 0)
            for (int o = 0; o < n; ++o) s += v[o * K + j];
        __syncthreads();
    }
    if (lr == 0) gt[(size_t)blockIdx.x * K + j] = s;
}

// a = (Gf^T Gf)^{-1} gt per column (gt = Gf^T x from k_gt_sum_multi), CTA per
// row: 64 entries of gt at a time are read by all threads and multiplied in
// order by thread j; alpha_out = -a when requested.  8 clusters, 32 load cases,
// alone: all rows in one CTA 23.7 us, one warp per row with its loads in
// rounds of 16 8.7 us, 4.5 us here.
__global__ void __launch_bounds__(256) k_gf_coef_multi(int K, int ncl, const double *__restrict__ invGtG,
                                                       const double *gt, double *a, double *alpha_out) {
    __shared__ double gs[64 * 32], is[64];
    pdl_next();
    const int m = 6 * ncl, q = blockIdx.x, j = threadIdx.x;
    if (j < min(64, m)) is[j] = invGtG[q + (size_t)j * m];
    pdl_wait();
    double s = 0.0;
    for (int p0 = 0; p0 < m; p0 += 64) {
        const int n = min(64, m - p0);
        if (p0 && j < n) is[j] = invGtG[q + (size_t)(p0 + j) * m];
#pragma unroll 8
        for (int o = j; o < n * K; o += 256) gs[o] = gt[(size_t)p0 * K + o];
        __syncthreads();
        if (j < K)
#pragma unroll 8
            for (int p = 0; p < n; ++p) s += is[p] * gs[p * K + j];
        __syncthreads();
    }
    if (j >= K) return;
    a[(size_t)q * K + j] = s;
    if (alpha_out) alpha_out[(size_t)q * K + j] = -s;
}

// largest values m of the columns over the CTA's 128 threads into xmax (FP32 bits, atomicMax)
__device__ __forceinline__ void col_max(double2 m, int K, unsigned *xmax) {
    __shared__ float red_max[256];
    red_max[2 * threadIdx.x] = (float)m.x;
    red_max[2 * threadIdx.x + 1] = (float)m.y;
    __syncthreads();
    if ((int)threadIdx.x < K) {
        float v = red_max[threadIdx.x];
        for (int t = threadIdx.x + K; t < 256; t += K) v = fmaxf(v, red_max[t]);
        if (v > 0.f) atomicMax(xmax + threadIdx.x, __float_as_uint(v));
    }
}

// Px = x - Gf a; partial dot with dotv per (block, j); blocks stride over
// row groups like k_rows_multi.  A row's clusters are read one step ahead, so
// that a step is one round of loads.
__global__ void __launch_bounds__(128) k_gf_apply_multi(int nlam, int K, const double *a, const int *__restrict__ gcl,
                                                        const double *__restrict__ gval, const double *x,
                                                        double *Px, const double *dotv, double *partial,
                                                        unsigned *xmax) {
    pdl_next();
    const int K2 = K / 2, lr = threadIdx.x / K2, j2 = threadIdx.x % K2;
    const int2 *cl = reinterpret_cast<const int2 *>(gcl);
    const double2 *x2 = reinterpret_cast<const double2 *>(x) + j2, *d2 = reinterpret_cast<const double2 *>(dotv) + j2;
    const double2 *a2 = reinterpret_cast<const double2 *>(a) + j2;
    double2 *p2 = reinterpret_cast<double2 *>(Px) + j2;
    const int stride = gridDim.x * (256 / K);
    int r = blockIdx.x * (256 / K) + lr;
    int2 c = make_int2(-1, -1);
    if (r < nlam) c = cl[r];
    pdl_wait();
    const double2 zero = make_double2(0.0, 0.0);
    double2 prod = zero, m = zero;
    for (; r < nlam; r += stride) {
        const int2 now = c;
        const double2 xv = x2[(size_t)r * K2], dv = dotv ? d2[(size_t)r * K2] : zero;
        if (r + stride < nlam) c = cl[r + stride];
        double2 v = zero;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int ck = k ? now.y : now.x;
            if (ck < 0) continue;
            const double2 *g = reinterpret_cast<const double2 *>(gval) + 3 * (size_t)(2 * r + k);
            const double2 *ac = a2 + 6 * ck * K2;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const double2 gq = g[q], a0 = ac[2 * q * K2], a1 = ac[(2 * q + 1) * K2];
                v.x += gq.x * a0.x;
                v.y += gq.x * a0.y;
                v.x += gq.y * a1.x;
                v.y += gq.y * a1.y;
            }
        }
        const double2 pv = make_double2(xv.x - v.x, xv.y - v.y);
        p2[(size_t)r * K2] = pv;
        m.x = fmax(m.x, fabs(pv.x));
        m.y = fmax(m.y, fabs(pv.y));
        if (dotv) {
            prod.x += pv.x * dv.x;
            prod.y += pv.y * dv.y;
        }
    }
    if (partial) block_col_partial(prod, K, partial);
    if (xmax) col_max(m, K, xmax);
}

// sum of partials of column j (fixed order), one CTA per column
__device__ double col_sum(const double *partial, int np, int K, int j) {
    __shared__ double red[256];
    double s = 0.0;
    for (int i = threadIdx.x; i < np; i += blockDim.x) s += partial[(size_t)i * K + j];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    const double r = red[0];
    __syncthreads();
    return r;
}

// per column: scalar = sum of partials -> out[j]; CTAs K .. 2 K - 1: of partial2 -> out2[j]; zero (2 K values, the
// column maxima) is set to zero on the way
__global__ void k_colsum(const double *partial, int np, int K, double *out, const double *partial2, double *out2,
                         unsigned *zero) {
    pdl_next();
    pdl_wait();
    const int j = blockIdx.x % K;
    const bool second = blockIdx.x >= K;
    const double s = col_sum(second ? partial2 : partial, np, K, j);
    if (threadIdx.x == 0) (second ? out2 : out)[j] = s;
    if (zero && blockIdx.x == 0 && threadIdx.x < 2 * K) zero[threadIdx.x] = 0;
}

// rho_j = -gPz_j / wFw_j ; lam += rho w ; g += rho Fw  (skips finished columns)
__global__ void __launch_bounds__(128) k_update_lam_g_multi(int n, int K, const double *wFw, const double *gw,
                                                            const double *w, const double *Fw,
                                                            double *lam, double *g, PcpgState *st) {
    pdl_next();
    pdl_wait();
    const long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x;      // pair of columns
    if (id >= (long long)n * (K / 2)) return;
    const int j = 2 * int(id % (K / 2));
    const bool run[2] = {!st[j].done, !st[j + 1].done};
    if (!run[0] && !run[1]) return;
    const double2 wv = reinterpret_cast<const double2 *>(w)[id], fv = reinterpret_cast<const double2 *>(Fw)[id];
    double2 lv = reinterpret_cast<double2 *>(lam)[id], gv = reinterpret_cast<double2 *>(g)[id];
    double rho[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        // mixed form: step length -g'w / w'Fw, equal to -g'Pz / w'Fw in exact
        // arithmetic and still the exact line minimum along w after the residual
        // g has been replaced by the FP64 one; FP64 form (no gw): -g'Pz / w'Fw
        const double d = wFw[j + k];
        rho[k] = -(gw ? gw[j + k] : st[j + k].gPz) / d;
        if (!(d > 0.0) || !isfinite(rho[k])) rho[k] = 0.0;
    }
    if (run[0]) {
        lv.x += rho[0] * wv.x;
        gv.x += rho[0] * fv.x;
    }
    if (run[1]) {
        lv.y += rho[1] * wv.y;
        gv.y += rho[1] * fv.y;
    }
    reinterpret_cast<double2 *>(lam)[id] = lv;
    reinterpret_cast<double2 *>(g)[id] = gv;
}

// w = Pz + gamma w (skips finished columns); with xmax also the column maxima of |w|, the scale of the next gather
__global__ void __launch_bounds__(128) k_update_w_multi(int n, int K, const double *gPz_new, const double *Pz,
                                                        double *w, const PcpgState *st, unsigned *xmax) {
    pdl_next();
    pdl_wait();
    const int stride = gridDim.x * 128, end = n * (K / 2);          // the stride is a multiple of K / 2
    const int id0 = blockIdx.x * 128 + threadIdx.x;
    const int j = 2 * (id0 % (K / 2));
    const bool run0 = !st[j].done, run1 = !st[j + 1].done;
    const double gam0 = run0 ? gPz_new[j] / st[j].gPz : 0.0, gam1 = run1 ? gPz_new[j + 1] / st[j + 1].gPz : 0.0;
    double2 *w2 = reinterpret_cast<double2 *>(w);
    const double2 *z2 = reinterpret_cast<const double2 *>(Pz);
    const double2 zero = make_double2(0.0, 0.0);
    double2 m = zero;
    for (long long id = id0; id < end; id += 2 * stride) {
        double2 v[2], z[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const bool here = id + u * stride < end;
            v[u] = here ? w2[id + u * stride] : zero;
            z[u] = here ? z2[id + u * stride] : zero;
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (run0) v[u].x = z[u].x + gam0 * v[u].x;
            if (run1) v[u].y = z[u].y + gam1 * v[u].y;
            if ((run0 || run1) && id + u * stride < end) w2[id + u * stride] = v[u];
            m.x = fmax(m.x, fabs(v[u].x));
            m.y = fmax(m.y, fabs(v[u].y));
        }
    }
    if (xmax) col_max(m, K, xmax);
}

// hist (FP64 form): relative residual of column j after iteration it at hist[it * K + j]
__global__ void k_finish_multi(int K, const double *wFw, const double *gPz_new,
                               PcpgState *st, double *hist) {
    pdl_next();
    pdl_wait();
    const int j = threadIdx.x;
    if (j >= K || st[j].done) return;
    const double gPz = gPz_new[j];
    st[j].wFw = wFw[j];
    st[j].gamma = gPz / st[j].gPz;
    st[j].gPz_prev = st[j].gPz;
    st[j].gPz = gPz;
    st[j].it += 1;
    st[j].rel = sqrt(gPz) / st[j].norm0;
    if (hist && st[j].it <= st[j].max_iter) hist[(size_t)st[j].it * K + j] = st[j].rel;
    if (!(wFw[j] > 0.0) || !isfinite(gPz)) st[j].done = 2;   // hand back to the FP64 residual check
    else if (sqrt(gPz) < st[j].eps * st[j].norm0) st[j].done = 1;
    else if (st[j].it >= st[j].max_iter) st[j].done = 3;
}

// strided column copy between a batch vector (stride K) and a plain vector
__global__ void k_col_get(int n, int K, int j, const double *__restrict__ B, double *__restrict__ v) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < n) v[r] = B[(size_t)r * K + j];
}
__global__ void k_col_set(int n, int K, int j, const double *__restrict__ v, double *__restrict__ B) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < n) B[(size_t)r * K + j] = v[r];
}

}  // namespace htf

namespace htf {

// ---------------------------------------------------------------------------
// FP64 residual of several load cases at once (the reliable-update step of
// the batched form): y_b(:, j) = A_d x_b(:, j) from the packed FP64 tiles for
// the K columns of a batch vector.  One CTA per (subdomain, 32-row block I)
// sums the tiles of block row I and, transposed, of block column I, so each
// output row is written once and no partial sums are needed.  The products
// run on the FP64 tensor path (mma.sync m8n8k4 .f64): warp w owns the 8-row
// band w mod 4 and K/16 column bands of 8; shared-memory row strides keep
// both operand loads free of bank conflicts.  With s given (the F apply),
// the coarse correction y_b -= V_d s_d is applied before the store.
// ---------------------------------------------------------------------------

// rows [32 I, 32 I + 32) of A X for the symmetric A of nt tile rows packed at
// base, X = x (RHS-interleaved, rows < nx; zero beyond): acc[q] = this
// thread's entries of row 8 band + g, columns 8 (cb0 + q) + 2 t4, + 1.  Tiles
// and X pieces are double-buffered in shared memory (one barrier each) and
// prefetched two ahead into registers; a tile above the diagonal is stored as
// it is and read transposed by the fragments.
template <int K>
__device__ __forceinline__ void sym_rows_product(const double *__restrict__ base, int nt, int I, const double *x,
                                                 int nx, double (&acc)[K / 16][2]) {
    constexpr int NT = K / 16;                      // 8x8 output tiles per warp
    constexpr int TS = 36, XS = K + 4;              // row strides (doubles): conflict-free fragment loads
    constexpr int TU = TILE_ELEMS / 256, XU = TILE * K / 256;
    __shared__ double Ts[2][32 * TS];
    __shared__ double Xs[2][32 * XS];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int g = lane >> 2, t4 = lane & 3;         // fragment row / column groups
    const int band = warp & 3, cb0 = (warp >> 2) * NT;
#pragma unroll
    for (int q = 0; q < NT; ++q) acc[q][0] = acc[q][1] = 0.0;
    double ta[TU], tb[TU], xa[XU], xc[XU];
    auto fetch_t = [&](double (&tr)[TU], int J) {
        const double *tp = base + (J <= I ? (long long)I * (I + 1) / 2 + J : (long long)J * (J + 1) / 2 + I) * TILE_ELEMS;
#pragma unroll
        for (int u = 0; u < TU; ++u) tr[u] = tp[threadIdx.x + 256 * u];
    };
    auto fetch_x = [&](double (&xr)[XU], int J) {
#pragma unroll
        for (int u = 0; u < XU; ++u) {
            const int e = threadIdx.x + 256 * u, r = TILE * J + e / K;
            xr[u] = r < nx ? x[(size_t)r * K + e % K] : 0.0;
        }
    };
    auto tile = [&](double (&tr)[TU], double (&xr)[XU], int J) {
        double *T = Ts[J & 1], *X = Xs[J & 1];
#pragma unroll
        for (int u = 0; u < TU; ++u) {
            const int e = threadIdx.x + 256 * u;
            T[(e / TILE) * TS + e % TILE] = tr[u];
        }
#pragma unroll
        for (int u = 0; u < XU; ++u) {
            const int e = threadIdx.x + 256 * u;
            X[(e / K) * XS + e % K] = xr[u];
        }
        __syncthreads();
        if (J + 2 < nt) {
            fetch_t(tr, J + 2);
            fetch_x(xr, J + 2);
        }
        const bool lower = J <= I;                  // tile (I, J): A[32I + r][32J + c]; else (J, I), transposed
        const double *Ta = T + (lower ? (8 * band + g) * TS + t4 : t4 * TS + 8 * band + g);
        const int step = lower ? 4 : 4 * TS;
#pragma unroll
        for (int kk = 0; kk < TILE / 4; ++kk) {
            const double a = Ta[kk * step];
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                const double bq = X[(4 * kk + t4) * XS + 8 * (cb0 + q) + g];
                dmma_8x8x4(acc[q][0], acc[q][1], a, bq);
            }
        }
    };
    pdl_next();
    fetch_t(ta, 0);
    if (nt > 1) fetch_t(tb, 1);
    pdl_wait();
    fetch_x(xa, 0);
    if (nt > 1) fetch_x(xc, 1);
    for (int J = 0; J < nt; J += 2) {
        tile(ta, xa, J);
        if (J + 1 < nt) tile(tb, xc, J + 1);
    }
}

template <int K>
__global__ void __launch_bounds__(256) k_symv_rows_multi(const int2 *__restrict__ rowblk,
                                                         const SubDev *__restrict__ subs,
                                                         const double *__restrict__ tiles,
                                                         const double *xb, double *yb,
                                                         const ClusterDev *__restrict__ cl,
                                                         const double *__restrict__ Vbuf,
                                                         const int *__restrict__ bcrows,
                                                         const double *s) {
    constexpr int NT = K / 16;
    const int2 rb = rowblk[blockIdx.x];
    const SubDev &sd = subs[rb.x];
    const int I = rb.y;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int g = lane >> 2, t4 = lane & 3;
    const int band = warp & 3, cb0 = (warp >> 2) * NT;
    double acc[NT][2];
    sym_rows_product<K>(tiles + sd.T_off * TILE_ELEMS, sd.nt, I, xb + (size_t)sd.xb_off * K, sd.nbp, acc);
    const int row = TILE * I + 8 * band + g;        // this thread's output row
    if (s && row < sd.nb) {
        const int gc_off = cl[sd.cluster].gc_off;
        const double *Vr = Vbuf + sd.V_off + row;
        for (int q = 0; q < sd.c + 6; ++q) {
            const double v = Vr[(size_t)q * sd.nbp];
            const int pos = q < sd.c ? bcrows[sd.bcr_off + q] : sd.alpha_pos + (q - sd.c);
            const double *sq = s + ((size_t)gc_off + pos) * K;
#pragma unroll
            for (int u = 0; u < NT; ++u) {
                const int col = 8 * (cb0 + u) + 2 * t4;
                acc[u][0] -= v * sq[col];
                acc[u][1] -= v * sq[col + 1];
            }
        }
    }
    double *y = yb + (size_t)(sd.xb_off + row) * K;
#pragma unroll
    for (int u = 0; u < NT; ++u) {
        const int col = 8 * (cb0 + u) + 2 * t4;
        y[col] = acc[u][0];
        y[col + 1] = acc[u][1];
    }
}
template __global__ void k_symv_rows_multi<16>(const int2 *, const SubDev *, const double *, const double *, double *,
                                               const ClusterDev *, const double *, const int *, const double *);
template __global__ void k_symv_rows_multi<32>(const int2 *, const SubDev *, const double *, const double *, double *,
                                               const ClusterDev *, const double *, const int *, const double *);

// S = M G per cluster from the packed symmetric tiles of M (pcpg_kernels.cu):
// CTA (cluster, 32-row block), the product of k_symv_rows_multi
template <int K>
__global__ void __launch_bounds__(256) k_msym_rows_multi(const int2 *__restrict__ mt,
                                                         const ClusterDev *__restrict__ cl,
                                                         const double *__restrict__ T, const double *gc,
                                                         double *s) {
    constexpr int NT = K / 16;
    const int2 b = mt[blockIdx.x];
    const ClusterDev c = cl[b.x];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int g = lane >> 2, t4 = lane & 3;
    const int band = warp & 3, cb0 = (warp >> 2) * NT;
    double acc[NT][2];
    sym_rows_product<K>(T + c.MT_off * TILE_ELEMS, c.mt, b.y, gc + (size_t)c.gc_off * K, c.ngc, acc);
    const int row = TILE * b.y + 8 * band + g;
    if (row >= c.ngc) return;
    double *y = s + (size_t)(c.gc_off + row) * K;
#pragma unroll
    for (int u = 0; u < NT; ++u) {
        const int col = 8 * (cb0 + u) + 2 * t4;
        y[col] = acc[u][0];
        y[col + 1] = acc[u][1];
    }
}
template __global__ void k_msym_rows_multi<16>(const int2 *, const ClusterDev *, const double *, const double *,
                                               double *);
template __global__ void k_msym_rows_multi<32>(const int2 *, const ClusterDev *, const double *, const double *,
                                               double *);

// B(:, j) = A(:, j) for the columns j with mask[j] (n rows, K-interleaved)
__global__ void k_cols_copy(long long n, int K, const int *__restrict__ mask, const double *__restrict__ A,
                            double *__restrict__ B) {
    for (long long o = blockIdx.x * (long long)blockDim.x + threadIdx.x; o < n * K;
         o += (long long)gridDim.x * blockDim.x)
        if (mask[o % K]) B[o] = A[o];
}

// per-column alpha (m values per column, column-major) of the columns with
// mask[j] from the projector's K-interleaved output
__global__ void k_alpha_cols(int m, int K, const int *__restrict__ mask, const double *a,
                             double *__restrict__ alpha) {
    for (int o = threadIdx.x; o < m * K; o += blockDim.x) {
        const int q = o / K, j = o % K;
        if (mask[j]) alpha[(size_t)j * m + q] = a[o];
    }
}

}  // namespace htf

// PCPG kernels of the HTFETI path (sm_100a), one load case.  All reductions
// are deterministic (fixed-order trees, no floating-point atomics), so a
// repeated solve gives the same bits.  (Load cases solved together go through
// pcpg_multi.cu, whose sums are grouped by its width: the same to round-off.)
//
//  F w = Bf K_HT^+ Bf^T w   (Cluster::mult_Ff, Cluster.cpp:1114-1188):
//    k_gather_b        x_b = Bf_d^T w             signed gather over the b slots
//    k_symv_units      y_b = F_d x_b              packed 32x32 lower tiles, one pass, in work
//                      t_d = V_d^T x_b            units; V = [F Bc_b^T, -R_b]
//    k_msym_rows       gc  = sum_d t_d            per cluster (gather map)
//    + k_msym_reduce   s   = M gc                 M = Ac^{-1} restricted, packed symmetric
//    k_reduce_correct  y_b = sum of the unit partials - V_d s_d
//    k_rows            Fw  = Bf y                 <= 2 entries per row
//  Preconditioner (Cluster::Preconditioning, Cluster.cpp:1043-1112):
//    k_gather_b(weighted) -> k_symv_units(S_d or K_bb) -> k_reduce_correct -> k_rows(weighted)
//  Projector (Cluster::Projection, Cluster.cpp:1314-1329):
//    k_gft_partial (Gf^T x per chunk, then a = (Gf^T Gf)^{-1} Gf^T x) -> k_gf_apply (x - Gf a)
#include <cuda_runtime.h>
#include <cstdint>

#include "device.cuh"

namespace htf {

constexpr unsigned FULL = 0xffffffffu;

// The kernels of one iteration run as a chain of programmatic dependent
// launches: a kernel lets its successor start as soon as all its own CTAs
// have started (pdl_next), and waits for its predecessor's results only where
// it first needs them (pdl_wait; every kernel of the chain waits, so a
// completed kernel implies all before it).  What does not change during a
// solve - tiles, gather lists, weights, Gf - is loaded before the wait, so a
// small problem's kernel costs one pass over the vectors it depends on instead
// of a launch plus a chain of dependent loads.  Pointers to data that the
// chain writes are not __restrict__, so that no load of them moves up.
// sum over the CTA's 256 threads in a fixed order (all threads get it); red: 8 doubles of shared memory
__device__ __forceinline__ double cta_sum(double v, double *red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    return ((red[0] + red[1]) + (red[2] + red[3])) + ((red[4] + red[5]) + (red[6] + red[7]));
}

// ---------------------------------------------------------------------------
// signed gather: x[slot] = sum_e sign_e * (weight[lam_e]) * w[lam_e]
// ent = 2*lam + (sign < 0)
// ---------------------------------------------------------------------------
__global__ void k_gather_b(int nslots, const int *__restrict__ ptr, const int *__restrict__ ent, const double *w,
                           const double *__restrict__ weight, double *x, const PcpgState *st) {
    pdl_next();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    int e0 = 0, e1 = 0, q[3];
    double wt[3];
    if (i < nslots) {
        e0 = ptr[i];
        e1 = ptr[i + 1];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {                   // a face slot has one entry, an edge slot three
        q[k] = e0 + k < e1 ? ent[e0 + k] : 0;
        wt[k] = weight && e0 + k < e1 ? weight[q[k] >> 1] : 1.0;
    }
    pdl_wait();
    if (i >= nslots || (st && st->done)) return;
    double v = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k)
        if (e0 + k < e1) {
            const double a = w[q[k] >> 1] * wt[k];
            v += (q[k] & 1) ? -a : a;
        }
    for (int e = e0 + 3; e < e1; ++e) {
        const int qe = ent[e], lam = qe >> 1;
        double a = w[lam];
        if (weight) a *= weight[lam];
        v += (qe & 1) ? -a : a;
    }
    x[i] = v;
}

// ---------------------------------------------------------------------------
// y_b = A x_b for packed symmetric tiles; one CTA per subdomain, 4 warps,
// per-warp partial sums in shared memory summed in fixed order.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void reduce_scatter32(double (&p)[32], int lane) {
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) {
        const bool upper = lane & s;
#pragma unroll
        for (int q = 0; q < s; ++q) {
            const double send = upper ? p[q] : p[q + s];
            const double keep = upper ? p[q + s] : p[q];
            p[q] = keep + __shfl_xor_sync(FULL, send, s);
        }
    }
}



// SYMV over work units (kinds 0 and 2) and V^T x (kind 1) in one launch; the
// partial y of a unit over its row window -> ypart[y_off, y_off + rows),
// summed later in unit order.  Shared memory: x and one partial y per warp
// over the unit's window.  A warp's first tile is loaded before the wait for
// x, its next one while the shuffles of the current one run.
__global__ void __launch_bounds__(SYMV_WARPS * 32) k_symv_units(const SymvUnit *__restrict__ units,
                                                                const SubDev *__restrict__ subs,
                                                                const double *__restrict__ tiles,
                                                                const double *__restrict__ Vbuf, const double *xb,
                                                                double *ypart, double *t, const PcpgState *st) {
    extern __shared__ double sm[];
    pdl_next();
    const SymvUnit u = units[blockIdx.x];
    const SubDev &sd = subs[u.d];
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    const double *x = xb + sd.xb_off;
    if (u.kind == 1) {                      // t_d = V_d^T x_b for columns [t0, t1), at most SYMV_VCOLS
        __shared__ double part[SYMV_WARPS][SYMV_VCOLS];
        const int c0 = int(u.t0), nc = int(u.t1 - u.t0), nb = sd.nb;
        const double *V = Vbuf + sd.V_off + (size_t)c0 * sd.nbp;
        const int t_off = sd.t_off + c0;
        const size_t nbp = sd.nbp;
        pdl_wait();
        if (st && st->done) return;
        double a[SYMV_VCOLS] = {};
#pragma unroll 2
        for (int i = threadIdx.x; i < nb; i += SYMV_WARPS * 32) {
            const double xi = x[i];
#pragma unroll
            for (int c = 0; c < SYMV_VCOLS; ++c) a[c] += (c < nc ? V[c * nbp + i] : 0.0) * xi;
        }
#pragma unroll
        for (int c = 0; c < SYMV_VCOLS; ++c) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a[c] += __shfl_xor_sync(FULL, a[c], o);
            if (lane == 0) part[warp][c] = a[c];
        }
        __syncthreads();
        if (threadIdx.x < nc) {
            double v = 0.0;
#pragma unroll
            for (int w = 0; w < SYMV_WARPS; ++w) v += part[w][threadIdx.x];
            t[t_off + threadIdx.x] = v;
        }
        return;
    }
    const int rows = u.rows, r0 = u.row0;
    // kind 0: window = rows [r0, r0 + rows); kind 2: rows [r0, r0 + seg) of the
    // column blocks, then the 32 rows of the unit's tile row at rowI
    const int seg = u.kind == 2 ? rows - TILE : rows;
    const double *base = tiles + sd.T_off * TILE_ELEMS;
    double v[32];
    long long tt = u.t0 + warp;
    if (tt < u.t1) {
        const double *tp = base + tt * TILE_ELEMS;
#pragma unroll
        for (int r = 0; r < 32; ++r) v[r] = tp[r * TILE + lane];
    }
    double *yp = sm + rows;                 // SYMV_WARPS x rows
    for (int i = threadIdx.x; i < SYMV_WARPS * rows; i += blockDim.x) yp[i] = 0.0;
    pdl_wait();
    if (st && st->done) return;
    for (int i = threadIdx.x; i < rows; i += blockDim.x) sm[i] = x[i < seg ? r0 + i : u.rowI + (i - seg)];
    __syncthreads();
    const double *xs = sm - r0;             // x of column block J at xs + 32 J
    double *ys = yp + warp * rows;          // this warp's partial y over the window
    double *my = ys - r0;                   // column block J at my + 32 J
    for (; tt < u.t1; tt += SYMV_WARPS) {
        int I = (int)((sqrt(8.0 * (double)tt + 1.0) - 1.0) * 0.5);
        while ((long long)(I + 1) * (I + 2) / 2 <= tt) ++I;
        while ((long long)I * (I + 1) / 2 > tt) --I;
        const int J = (int)(tt - (long long)I * (I + 1) / 2);
        const double xJ = xs[TILE * J + lane];
        const double *xI = u.kind == 2 ? sm + seg : xs + TILE * I;      // x of row block I
        double *yI = u.kind == 2 ? ys + seg : my + TILE * I;             // partial y of row block I
        double p[32];
        double col = 0.0;
#pragma unroll
        for (int r = 0; r < 32; ++r) {
            p[r] = v[r] * xJ;
            col += v[r] * xI[r];
        }
        if (tt + SYMV_WARPS < u.t1) {
            const double *tp = base + (tt + SYMV_WARPS) * TILE_ELEMS;
#pragma unroll
            for (int r = 0; r < 32; ++r) v[r] = tp[r * TILE + lane];
        }
        reduce_scatter32(p, lane);
        yI[lane] += p[0];
        if (I != J) my[TILE * J + lane] += col;
    }
    __syncthreads();
    double *out = ypart + u.y_off;
    for (int i = threadIdx.x; i < rows; i += blockDim.x) {
        double a = 0.0;
#pragma unroll
        for (int q = 0; q < SYMV_WARPS; ++q) a += yp[q * rows + i];
        out[i] = a;
    }
}

// y_b = sum of the unit partials [- V_d s_d with CORRECT].  CTA
// (subdomain, 64 b rows) of four groups of 64 threads: thread (group k, row)
// adds the partials k, k + 4, .. of the row's block (rboff: where each
// unit's 32 partial rows of the block start in ypart, in unit order) and the
// columns k, k + 4, .. of V; the groups are added in order.  V's first
// RC_PRE columns of a thread and the lists are loaded before the wait.
// Bound by latency (a large subdomain has some 50 partials a row).  Without the
// correction a warp, whose 32 rows share their block's list, reads up to 32
// offsets at once, before the wait, and keeps eight partials in flight: S_i of
// the 512-subdomain cube 34 -> 28 us, of 4 096 uneven subdomains 346 -> 292.
// With V's columns in flight too that costs the registers of a CTA per SM (55
// -> 58 and 540 -> 598 us), so F_i reads each offset before its partial.
template <bool CORRECT>
__global__ void __launch_bounds__(256) k_reduce_correct(const SubDev *__restrict__ subs,
                                                        const int *__restrict__ rbptr,
                                                        const long long *__restrict__ rboff, const double *ypart,
                                                        const ClusterDev *__restrict__ cl,
                                                        const double *__restrict__ Vbuf,
                                                        const int *__restrict__ bcrows, const double *s, double *yb,
                                                        const PcpgState *st) {
    constexpr int RC_PRE = 8, U = 8;
    __shared__ double sd_s[CORRECT ? 256 : 1];
    __shared__ double part[3][64];
    pdl_next();
    const SubDev &sd = subs[blockIdx.x];
    const int grp = threadIdx.x >> 6, lr = threadIdx.x & 63, i = blockIdx.y * 64 + lr, lane = threadIdx.x & 31;
    if (blockIdx.y * 64 >= sd.nbp) return;
    const bool in = i < sd.nbp;             // nbp is a multiple of 32, not of 64: the same for a warp
    const int nc = CORRECT ? sd.c + 6 : 0;
    const double *V = Vbuf + sd.V_off + i;
    const size_t nbp = sd.nbp;
    const int q0 = in ? rbptr[sd.rb_off + i / TILE] : 0, q1 = in ? rbptr[sd.rb_off + i / TILE + 1] : 0;
    long long off = !CORRECT && q0 + grp + 4 * lane < q1 ? rboff[q0 + grp + 4 * lane] : 0;
    double vr[RC_PRE];
    int pos = -1;
    if (CORRECT) {
#pragma unroll
        for (int u = 0; u < RC_PRE; ++u) vr[u] = (in && grp + 4 * u < nc) ? V[(grp + 4 * u) * nbp] : 0.0;
        if (int(threadIdx.x) < nc)
            pos = cl[sd.cluster].gc_off +
                  (int(threadIdx.x) < sd.c ? bcrows[sd.bcr_off + threadIdx.x] : sd.alpha_pos + (int(threadIdx.x) - sd.c));
    }
    pdl_wait();
    if (st && st->done) return;
    if (CORRECT && pos >= 0) sd_s[threadIdx.x] = s[pos];           // c + 6 <= 256
    double a = 0.0;
    if (CORRECT) {
#pragma unroll 4
        for (int q = q0 + grp; q < q1; q += 4) a += ypart[rboff[q] + lane];
    } else {
        for (int q = q0 + grp; q < q1; q += 4 * 32) {              // 32 partials of this group at a time
            if (q != q0 + grp) off = q + 4 * lane < q1 ? rboff[q + 4 * lane] : 0;
            const int n = min(32, (q1 - q + 3) / 4);
            for (int k = 0; k < n; k += U) {
                double v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const long long o = __shfl_sync(FULL, off, (k + u) & 31);
                    v[u] = k + u < n ? ypart[o + lane] : 0.0;
                }
#pragma unroll
                for (int u = 0; u < U; ++u) a += v[u];
            }
        }
    }
    if (CORRECT) {
        __syncthreads();
        double b = 0.0;
#pragma unroll
        for (int u = 0; u < RC_PRE; ++u) b += (grp + 4 * u < nc) ? vr[u] * sd_s[grp + 4 * u] : 0.0;
        if (in)
#pragma unroll 4
            for (int q = grp + 4 * RC_PRE; q < nc; q += 4) b += V[q * nbp] * sd_s[q];
        a -= b;
    }
    if (grp) part[grp - 1][lr] = a;
    __syncthreads();
    if (grp == 0 && in) yb[sd.xb_off + i] = ((a + part[0][lr]) + part[1][lr]) + part[2][lr];
}
template __global__ void k_reduce_correct<false>(const SubDev *, const int *, const long long *, const double *,
                                                 const ClusterDev *, const double *, const int *, const double *,
                                                 double *, const PcpgState *);
template __global__ void k_reduce_correct<true>(const SubDev *, const int *, const long long *, const double *,
                                                const ClusterDev *, const double *, const int *, const double *,
                                                double *, const PcpgState *);

// gc[q] = sum of the t entries listed for q (fixed order)
__global__ void k_gc(int ngc_total, const int *__restrict__ gptr, const int *__restrict__ gidx,
                     const double *__restrict__ t, double *__restrict__ gc, const PcpgState *__restrict__ st) {
    if (st && st->done) return;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= ngc_total) return;
    double s = 0.0;
    for (int e = gptr[q]; e < gptr[q + 1]; ++e) s += t[gidx[e]];
    gc[q] = s;
}

// s = M gc per cluster; one warp per row
__global__ void k_coarse(const ClusterDev *__restrict__ cl, const double *__restrict__ Mbuf,
                         const double *__restrict__ gc, double *__restrict__ s, const PcpgState *__restrict__ st) {
    if (st && st->done) return;
    const ClusterDev c = cl[blockIdx.x];
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32, nw = blockDim.x / 32;
    const int row = blockIdx.y * nw + warp;
    if (row >= c.ngc) return;
    const double *M = Mbuf + c.M_off + (size_t)row * c.ngc;     // symmetric: column = row
    const double *g = gc + c.gc_off;
    double a = 0.0;
    for (int p = lane; p < c.ngc; p += 32) a += M[p] * g[p];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(FULL, a, o);
    if (lane == 0) s[c.gc_off + row] = a;
}

// y_b -= V_d s_d  with s_d = (s at the Bc rows of d, alpha_d)
__global__ void k_correct(const SubDev *__restrict__ subs, const ClusterDev *__restrict__ cl,
                          const double *__restrict__ Vbuf, const int *__restrict__ bcrows,
                          const double *__restrict__ s, double *__restrict__ yb, const PcpgState *__restrict__ st) {
    if (st && st->done) return;
    __shared__ double sd_s[256];
    const SubDev &sd = subs[blockIdx.x];
    const ClusterDev &c = cl[sd.cluster];
    const int nc = sd.c + 6;
    for (int q = threadIdx.x; q < nc; q += blockDim.x) {
        const int pos = (q < sd.c) ? bcrows[sd.bcr_off + q] : sd.alpha_pos + (q - sd.c);
        sd_s[q] = s[c.gc_off + pos];
    }
    __syncthreads();
    const double *V = Vbuf + sd.V_off;
    double *y = yb + sd.xb_off;
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < sd.nb; i += gridDim.y * blockDim.x) {
        double a = y[i];
#pragma unroll 8
        for (int q = 0; q < nc; ++q) a -= V[i + (size_t)q * sd.nbp] * sd_s[q];
        y[i] = a;
    }
}

// out[r] = wt[r] * sum_k sign_k * y[slot_k]; optional fused dot partial with `dotv`
__global__ void __launch_bounds__(256) k_rows(int nlam, const int *__restrict__ rslot,
                                              const double *__restrict__ rsign, const double *yb,
                                              const double *__restrict__ weight, double *out, const double *dotv,
                                              double *partial, const PcpgState *st) {
    __shared__ double red[8];
    pdl_next();
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    int2 sl = make_int2(-1, -1);
    double2 sg = make_double2(0.0, 0.0);
    double wt = 1.0;
    if (r < nlam) {
        sl = reinterpret_cast<const int2 *>(rslot)[r];
        sg = reinterpret_cast<const double2 *>(rsign)[r];
        if (weight) wt = weight[r];
    }
    pdl_wait();
    if (st && st->done) return;
    double prod = 0.0;
    if (r < nlam) {
        double v = 0.0;
        if (sl.x >= 0) v += sg.x * yb[sl.x];
        if (sl.y >= 0) v += sg.y * yb[sl.y];
        v *= wt;
        out[r] = v;
        if (dotv) prod = v * dotv[r];
    }
    if (!partial) return;
    const double sum = cta_sum(prod, red);
    if (threadIdx.x == 0) partial[blockIdx.x] = sum;
}

// sum of np partials in a fixed order, by every CTA (256 threads)
__device__ __forceinline__ double block_sum_fixed(const double *partial, int np, double *red) {
    double s = 0.0;
#pragma unroll 4
    for (int i = threadIdx.x; i < np; i += 256) s += partial[i];
    return cta_sum(s, red);
}

// ---------------------------------------------------------------------------
// projector: a = (Gf^T Gf)^{-1} Gf^T x ; Px = x - Gf a
// Gf stored per cluster as a list of (row, 6 values) cut into chunks of up to
// 1024 rows; per row as up to two (cluster, 6 values) entries.
//
// In the iteration x is the updated residual g + rho Fw (Cluster::pcpg,
// Cluster.cpp:1426-1430): k_gft_partial forms it where it reads g, and
// k_gf_apply, which visits every row once, writes g and lambda back.
//
// k_gft_partial: CTA ch sums its chunk's six products; the CTA that finishes
// last (a counter, which it sets back to zero) adds the chunks of every
// cluster, multiplies by (Gf^T Gf)^{-1} and writes a (and -a), both in a
// fixed order whichever CTA that is.  a may be the partials' own array: all of
// them have been read by then.
// ---------------------------------------------------------------------------
// rho = -gPz / wFw from the partials of w.Fw (256 threads; every CTA the same value)
__device__ __forceinline__ double step_length(const double *partial, int np, double *red, const PcpgState *st,
                                              double &wFw) {
    const double gPz = st->gPz;
    wFw = block_sum_fixed(partial, np, red);
    const double rho = -gPz / wFw;
    return (!(wFw > 0.0) || !isfinite(rho)) ? 0.0 : rho;
}

__global__ void __launch_bounds__(256) k_gft_partial(const int *__restrict__ chunk_beg,
                                                     const int *__restrict__ chunk_end,
                                                     const int *__restrict__ crow, const double *__restrict__ cval,
                                                     const double *x, double *partial, int ncl,
                                                     const int *__restrict__ cl_chunk_ptr,
                                                     const double *__restrict__ invGtG, double *a_out,
                                                     double *alpha_out, unsigned *counter, const double *Fw,
                                                     const double *wFw_part, int np, PcpgState *st) {
    extern __shared__ double gt[];                  // 6 ncl
    __shared__ double red[8][6];
    __shared__ double red8[8];
    __shared__ bool last;
    pdl_next();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int beg = chunk_beg[blockIdx.x], end = chunk_end[blockIdx.x];
    // up to 1024 rows: four per thread, loaded before the wait
    int row[4];
    double g[4][6];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int e = beg + int(threadIdx.x) + 256 * k;
        row[k] = e < end ? crow[e] : -1;
        const double2 *c = reinterpret_cast<const double2 *>(cval + 6 * (size_t)e);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const double2 d = e < end ? c[q] : make_double2(0.0, 0.0);
            g[k][2 * q] = d.x;
            g[k][2 * q + 1] = d.y;
        }
    }
    pdl_wait();
    if (st && st->done) return;
    double xr[4], fr[4], rho = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        xr[k] = row[k] >= 0 ? x[row[k]] : 0.0;
        fr[k] = Fw && row[k] >= 0 ? Fw[row[k]] : 0.0;
    }
    if (Fw) {
        double wFw;
        rho = step_length(wFw_part, np, red8, st, wFw);
    }
    double s[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double xv = Fw ? xr[k] + rho * fr[k] : xr[k];
#pragma unroll
        for (int q = 0; q < 6; ++q) s[q] += g[k][q] * xv;
    }
#pragma unroll
    for (int q = 0; q < 6; ++q) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[q] += __shfl_xor_sync(FULL, s[q], o);
        if (lane == 0) red[warp][q] = s[q];
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) v += red[w][threadIdx.x];
        partial[6 * (size_t)blockIdx.x + threadIdx.x] = v;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
        if (last) *counter = 0;
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    const int m = 6 * ncl;
    for (int q = warp; q < m; q += 8) {             // one warp per (cluster, mode)
        const int c = q / 6, i = q % 6;
        double v = 0.0;
#pragma unroll 4
        for (int ch = cl_chunk_ptr[c] + lane; ch < cl_chunk_ptr[c + 1]; ch += 32)
            v += __ldcg(partial + 6 * (size_t)ch + i);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
        if (lane == 0) gt[q] = v;
    }
    __syncthreads();
    for (int q = warp; q < m; q += 8) {
        double v = 0.0;
        for (int p = lane; p < m; p += 32) v += invGtG[q + (size_t)p * m] * gt[p];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
        if (lane == 0) {
            a_out[q] = v;
            if (alpha_out) alpha_out[q] = -v;
        }
    }
}

// Px = x - Gf a for the coefficient a of k_gft_partial (and the partials of Px.dotv)
__global__ void __launch_bounds__(256) k_gf_apply(int nlam, int ncl, const double *acoef,
                                                  const int *__restrict__ gcl, const double *__restrict__ gval,
                                                  const double *x, double *Px, const double *dotv, double *partial,
                                                  unsigned *reset, const double *w, const double *Fw,
                                                  const double *wFw_part, int np, double *lam, double *g_out,
                                                  PcpgState *st) {
    extern __shared__ double sh[];
    double *a = sh;                  // 6*ncl
    __shared__ double red[8];
    pdl_next();
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    int2 c = make_int2(-1, -1);
    double2 g[6];
    if (r < nlam) {
        c = reinterpret_cast<const int2 *>(gcl)[r];
        const double2 *gp = reinterpret_cast<const double2 *>(gval + 12 * (size_t)r);
#pragma unroll
        for (int q = 0; q < 6; ++q) g[q] = gp[q];
    }
    pdl_wait();
    if (st && st->done) return;
    if (reset && blockIdx.x == 0 && threadIdx.x == 0) *reset = 0;
    for (int q = threadIdx.x; q < 6 * ncl; q += blockDim.x) a[q] = acoef[q];
    double xr = r < nlam ? x[r] : 0.0;
    if (Fw) {                                        // lam += rho w ; g += rho Fw (x is g)
        const double fw = r < nlam ? Fw[r] : 0.0, wr = r < nlam ? w[r] : 0.0, lr = r < nlam ? lam[r] : 0.0;
        double wFw;
        const double rho = step_length(wFw_part, np, red, st, wFw);
        if (r < nlam) {
            xr += rho * fw;
            g_out[r] = xr;
            lam[r] = lr + rho * wr;
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            st->wFw = wFw;
            st->rho = rho;
        }
    }
    __syncthreads();
    double prod = 0.0;
    if (r < nlam) {
        double v = 0.0;
        if (c.x >= 0)
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                v += g[q].x * a[6 * c.x + 2 * q];
                v += g[q].y * a[6 * c.x + 2 * q + 1];
            }
        if (c.y >= 0)
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                v += g[3 + q].x * a[6 * c.y + 2 * q];
                v += g[3 + q].y * a[6 * c.y + 2 * q + 1];
            }
        const double pv = xr - v;
        Px[r] = pv;
        if (dotv) prod = pv * dotv[r];
    }
    if (!partial) return;
    const double sum = cta_sum(prod, red);
    if (threadIdx.x == 0) partial[blockIdx.x] = sum;
}

// lambda = G a  (initial lambda0 = Gf (GfTGf)^{-1} e)
__global__ void k_gf_mult(int nlam, const int *__restrict__ gcl, const double *__restrict__ gval,
                          const double *__restrict__ a, double *__restrict__ out) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nlam) return;
    double v = 0.0;
    for (int k = 0; k < 2; ++k) {
        const int c = gcl[2 * r + k];
        if (c < 0) continue;
        const double *g = gval + 6 * (size_t)(2 * r + k);
        for (int q = 0; q < 6; ++q) v += g[q] * a[6 * c + q];
    }
    out[r] = v;
}

// ---------------------------------------------------------------------------
// PCPG scalar / vector updates (Cluster::pcpg, Cluster.cpp:1422-1450)
// ---------------------------------------------------------------------------
// after Fw and the partials of w.Fw: rho = -gPz / wFw ; lam += rho w ; g += rho Fw
// (problems of more rows than the projector updates on the way)
__global__ void __launch_bounds__(256) k_update_lam_g(int n, const double *partial, int np, const double *w,
                                                      const double *Fw, double *lam, double *g, PcpgState *st) {
    __shared__ double red[8];
    pdl_next();
    pdl_wait();
    if (st->done) return;
    double wFw;
    const double rho = step_length(partial, np, red, st, wFw);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->wFw = wFw;
        st->rho = rho;
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        lam[i] += rho * w[i];
        g[i] += rho * Fw[i];
    }
}

// after Pz and the partials of g.Pz: gamma = gPz / (gPz before), w = Pz +
// gamma w.  The CTA that finishes last (counter, set back to zero) commits
// the iteration: gPz and gamma, the count, the convergence test, and the
// relative residual sqrt(g'Pz)/sqrt(g0'Pz0) of iteration it in hist[it]
// (nhist entries: a state set up for timing may run past them).
__global__ void __launch_bounds__(256) k_update_w(int n, const double *partial, int np, const double *Pz, double *w,
                                                  PcpgState *st, double *hist, int nhist, unsigned *counter) {
    __shared__ double red[8];
    pdl_next();
    pdl_wait();
    if (st->done) return;
    const double old = st->gPz;
    const double gPz = block_sum_fixed(partial, np, red);
    const double gam = gPz / old;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) w[i] = Pz[i] + gam * w[i];
    __syncthreads();                                 // every thread has read the state
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(counter, 1u) == gridDim.x - 1) {
            *counter = 0;
            st->gamma = gam;
            st->gPz_prev = old;
            st->gPz = gPz;
            st->it += 1;
            st->rel = sqrt(gPz) / st->norm0;
            if (st->it < nhist) hist[st->it] = st->rel;
            if (!(st->wFw > 0.0) || !isfinite(gPz)) st->done = 2;          // breakdown
            else if (sqrt(gPz) < st->eps * st->norm0) st->done = 1;        // converged
            else if (st->it >= st->max_iter) st->done = 3;                  // max_iter
        }
    }
}

// initial state: norm0 = sqrt(g0.Pz0)
__global__ void k_init_state(const double *__restrict__ partial, int np, PcpgState *__restrict__ st, double eps,
                             int max_iter) {
    __shared__ double red[8];
    const double gPz = block_sum_fixed(partial, np, red);
    if (threadIdx.x == 0) {
        st->gPz = gPz;
        st->gPz_prev = gPz;
        st->norm0 = sqrt(gPz);
        st->rel = 1.0;
        st->it = 0;
        st->eps = eps;
        st->max_iter = max_iter;
        st->wFw = 1.0;
        st->done = (gPz > 0.0 && isfinite(gPz)) ? ((max_iter <= 0) ? 3 : 0) : (gPz == 0.0 ? 1 : 2);
    }
}

// generic: y = a*x + b*y on n entries
__global__ void k_axpby(int n, double a, const double *__restrict__ x, double b, double *__restrict__ y) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = a * x[i] + b * y[i];
}

// ---------------------------------------------------------------------------
// Dirichlet preconditioner without the dense S_d (preconditioner =
// Dirichlet_implicit, the reference's Cluster.cpp:1082-1104 variant that
// keeps no explicit S_d): the factor of K_reg,d eliminates the interior
// first, so its trailing b-set columns hold L_bb with L_bb L_bb^T = S_reg =
// S_d + D_fix (D_fix = the original diagonal at the 6 fix DOFs).  y_b =
// S_d x_b = L_bb (L_bb^T x_b) - D_fix x_b, two passes over the b-set
// column panels of the resident factor, no S_d stored.
//   k_lbt_x: t = L_bb^T x_b, one CTA per (subdomain, 32-column block p):
//            4 warps over the 32-row blocks R >= p, lane l row 32 R + l,
//            32 column sums per lane, reduce-scatter, warps added in order;
//   k_lb_t:  y = L_bb t - D_fix x_b, one CTA per (subdomain, 32-row block R):
//            4 warps over the column blocks p <= R, warps added in order.
// Each block of L_bb is read once per pass, 32 contiguous rows of a column
// per warp load.  `blk` lists (subdomain, block) pairs.
// ---------------------------------------------------------------------------
__global__ void k_lbt_x(const int2 *__restrict__ blk, const SubDev *__restrict__ subs, const double *__restrict__ K,
                        const double *xb, double *tb, const PcpgState *st) {
    __shared__ double part[4][32];
    pdl_next();
    const int2 b = blk[blockIdx.x];
    const SubDev sd = subs[b.x];
    const int p = b.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cb = sd.nr + 32 * p;
    double acc[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) acc[j] = 0.0;
    // the 32 columns are one factor panel: (r, cb + j) at pbase + j * ld + r
    const double *pbase = K + kcol(sd, cb);
    const long long ld = kld(sd, cb);
    double l[32];
    auto load = [&](int R) {
        const double *col = pbase + sd.nr + 32 * R + lane;
#pragma unroll
        for (int j = 0; j < 32; ++j) l[j] = (R > p || lane >= j) ? col[j * ld] : 0.0;
    };
    if (p + warp < sd.nt) load(p + warp);
    pdl_wait();
    if (st && st->done) return;
    for (int R = p + warp; R < sd.nt; R += 4) {
        const double xr = xb[sd.xb_off + 32 * R + lane];
#pragma unroll
        for (int j = 0; j < 32; ++j) acc[j] += l[j] * xr;
        if (R + 4 < sd.nt) load(R + 4);
    }
    reduce_scatter32(acc, lane);
    part[warp][lane] = acc[0];
    __syncthreads();
    if (warp == 0)
        tb[sd.xb_off + 32 * p + lane] = ((part[0][lane] + part[1][lane]) + part[2][lane]) + part[3][lane];
}

__global__ void k_lb_t(const int2 *__restrict__ blk, const SubDev *__restrict__ subs, const double *__restrict__ K,
                       const double *tb, const double *xb, double *yb, const PcpgState *st) {
    __shared__ double part[4][32];
    pdl_next();
    const int2 b = blk[blockIdx.x];
    const SubDev sd = subs[b.x];
    const int R = b.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = sd.nr + 32 * R + lane;
    double z = 0.0, l[32];
    auto load = [&](int p) {
        const int cb = sd.nr + 32 * p;
        const double *col = K + kcol(sd, cb) + r;      // (r, cb + j) at col + j * ld
        const long long ld = kld(sd, cb);
#pragma unroll
        for (int j = 0; j < 32; ++j) l[j] = (p < R || lane >= j) ? col[j * ld] : 0.0;
    };
    if (warp <= R) load(warp);
    pdl_wait();
    if (st && st->done) return;
    for (int p = warp; p <= R; p += 4) {
        const double tl = tb[sd.xb_off + 32 * p + lane];
#pragma unroll
        for (int j = 0; j < 32; ++j) z += l[j] * __shfl_sync(FULL, tl, j);
        if (p + 4 <= R) load(p + 4);
    }
    part[warp][lane] = z;
    __syncthreads();
    if (warp == 0) {
        double y = ((part[0][lane] + part[1][lane]) + part[2][lane]) + part[3][lane];
#pragma unroll
        for (int k = 0; k < 6; ++k)
            if (sd.fix[k] == r) y -= sd.fix_diag[k] * xb[sd.xb_off + 32 * R + lane];
        yb[sd.xb_off + 32 * R + lane] = y;
    }
}

// ---------------------------------------------------------------------------
// Coarse solve s = M gc with the symmetric M stored once, as packed lower
// 32x32 tiles (tile (I, J), J <= I, at MT_off + I (I + 1) / 2 + J, row-major
// inside, diagonal tiles full): half the bytes of the dense M every F apply
// reads.  `mt` lists (cluster, tile row) pairs.
//   k_pack_M:      tiles of tile row I from the dense M (set-up);
//   k_msym_rows:   CTA (cluster, I), 4 warps over the tiles of row I, the
//                  coarse right-hand side gc summed from the subdomains' t
//                  on the way: the direct product M_IJ x_J summed per warp
//                  then in warp order into D[I]; the transposed M_IJ^T x_I
//                  (J < I) of each tile into its own 32-value slot P[(I, J)];
//   k_msym_reduce: s_J = D[J] + sum over I > J of P[(I, J)]: warp w every
//                  fourth I from J + 1 + w, the warps added in order.
// Every tile is read once and every sum has a fixed order.
// ---------------------------------------------------------------------------
__global__ void k_pack_M(const int2 *__restrict__ mt, const ClusterDev *__restrict__ cl,
                         const double *__restrict__ M, double *__restrict__ T) {
    const int2 b = mt[blockIdx.x];
    const ClusterDev c = cl[b.x];
    const int I = b.y;
    double *row = T + (c.MT_off + (long long)I * (I + 1) / 2) * TILE_ELEMS;
    for (int idx = threadIdx.x; idx < (I + 1) * TILE_ELEMS; idx += blockDim.x) {
        const int J = idx / TILE_ELEMS, e = idx % TILE_ELEMS, r = e / TILE, j = e % TILE;
        const int gr = TILE * I + r, gcn = TILE * J + j;
        row[idx] = (gr < c.ngc && gcn < c.ngc) ? M[c.M_off + gr + (size_t)gcn * c.ngc] : 0.0;
    }
}

__global__ void __launch_bounds__(128) k_msym_rows(const int2 *__restrict__ mt, const ClusterDev *__restrict__ cl,
                                                   const double *__restrict__ T, const int *__restrict__ gptr,
                                                   const int *__restrict__ gidx, const double *t, double *D, double *P,
                                                   const PcpgState *st) {
    __shared__ double xI[TILE];
    __shared__ double part[4][TILE];
    pdl_next();
    const int2 b = mt[blockIdx.x];
    const ClusterDev c = cl[b.x];
    const int I = b.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long t0 = c.MT_off + (long long)I * (I + 1) / 2;
    double v[32];
    // tile J of this row and the t entries behind its column's coarse right-hand side: loaded before the wait,
    // then while the previous tile is summed
    int e0 = 0, e1 = 0, i0 = 0, i1 = 0;
    auto load = [&](int J) {
        const double *tp = T + (t0 + J) * TILE_ELEMS;
#pragma unroll
        for (int r = 0; r < 32; ++r) v[r] = tp[r * TILE + lane];
        e0 = e1 = 0;
        const int q = TILE * J + lane;
        if (q < c.ngc) {
            e0 = gptr[c.gc_off + q];
            e1 = gptr[c.gc_off + q + 1];
        }
        i0 = e0 < e1 ? gidx[e0] : 0;
        i1 = e0 + 1 < e1 ? gidx[e0 + 1] : 0;
    };
    auto rhs = [&] {                        // gc[q] = sum of the t entries listed for q, in list order
        double g = e0 < e1 ? t[i0] : 0.0;
        if (e0 + 1 < e1) g += t[i1];
        for (int e = e0 + 2; e < e1; ++e) g += t[gidx[e]];
        return g;
    };
    if (warp == 0) {
        const int q = TILE * I + lane;
        int f0 = 0, f1 = 0;
        if (q < c.ngc) {
            f0 = gptr[c.gc_off + q];
            f1 = gptr[c.gc_off + q + 1];
        }
        const int k0 = f0 < f1 ? gidx[f0] : 0, k1 = f0 + 1 < f1 ? gidx[f0 + 1] : 0;
        load(0);
        pdl_wait();
        double g = f0 < f1 ? t[k0] : 0.0;
        if (f0 + 1 < f1) g += t[k1];
        for (int e = f0 + 2; e < f1; ++e) g += t[gidx[e]];
        xI[lane] = g;
    } else {
        if (warp <= I) load(warp);
        pdl_wait();
    }
    if (st && st->done) return;
    __syncthreads();
    double dir = 0.0;
    for (int J = warp; J <= I; J += 4) {
        const double xJ = rhs();
        double p[32];
        double col = 0.0;
#pragma unroll
        for (int r = 0; r < 32; ++r) {
            p[r] = v[r] * xJ;
            col += v[r] * xI[r];
        }
        if (J + 4 <= I) load(J + 4);
        reduce_scatter32(p, lane);
        dir += p[0];
        if (J < I) P[(t0 + J) * TILE + lane] = col;
    }
    part[warp][lane] = dir;
    __syncthreads();
    if (warp == 0)
        D[((long long)c.mt_row_off + I) * TILE + lane] = ((part[0][lane] + part[1][lane]) + part[2][lane]) + part[3][lane];
}

// Both in one launch for a small M: CTA (cluster, J) reads the tiles of row J
// and, transposed, of column J (every off-diagonal tile twice, the second
// time from L2), with the sums of the two kernels in the same order.
__global__ void __launch_bounds__(128) k_msym_small(const int2 *__restrict__ mt, const ClusterDev *__restrict__ cl,
                                                    const double *__restrict__ T, const int *__restrict__ gptr,
                                                    const int *__restrict__ gidx, const double *t, double *s,
                                                    const PcpgState *st) {
    __shared__ double part[4][TILE];
    __shared__ double xs[4][TILE];
    pdl_next();
    const int2 b = mt[blockIdx.x];
    const ClusterDev c = cl[b.x];
    const int J = b.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double v[32];
    int e0 = 0, e1 = 0, i0 = 0, i1 = 0;
    // tile (A, B), A >= B, and the t entries behind the coarse right-hand side of block X
    auto load = [&](int A, int B, int X) {
        const double *tp = T + (c.MT_off + (long long)A * (A + 1) / 2 + B) * TILE_ELEMS;
#pragma unroll
        for (int r = 0; r < 32; ++r) v[r] = tp[r * TILE + lane];
        e0 = e1 = 0;
        const int q = TILE * X + lane;
        if (q < c.ngc) {
            e0 = gptr[c.gc_off + q];
            e1 = gptr[c.gc_off + q + 1];
        }
        i0 = e0 < e1 ? gidx[e0] : 0;
        i1 = e0 + 1 < e1 ? gidx[e0 + 1] : 0;
    };
    auto rhs = [&] {
        double g = e0 < e1 ? t[i0] : 0.0;
        if (e0 + 1 < e1) g += t[i1];
        for (int e = e0 + 2; e < e1; ++e) g += t[gidx[e]];
        return g;
    };
    if (warp <= J) load(J, warp, warp);
    pdl_wait();
    if (st && st->done) return;
    double dir = 0.0;
    for (int B = warp; B <= J; B += 4) {
        const double xB = rhs();
        double p[32];
#pragma unroll
        for (int r = 0; r < 32; ++r) p[r] = v[r] * xB;
        if (B + 4 <= J) load(J, B + 4, B + 4);
        reduce_scatter32(p, lane);
        dir += p[0];
    }
    part[warp][lane] = dir;
    __syncthreads();
    double y = warp == 0 ? ((part[0][lane] + part[1][lane]) + part[2][lane]) + part[3][lane] : 0.0;
    __syncthreads();
    for (int I = J + 1 + warp; I < c.mt; I += 4) {
        load(I, J, I);
        xs[warp][lane] = rhs();
        __syncwarp();
        double col = 0.0;
#pragma unroll
        for (int r = 0; r < 32; ++r) col += v[r] * xs[warp][r];
        __syncwarp();
        y += col;
    }
    part[warp][lane] = y;
    __syncthreads();
    if (warp == 0 && TILE * J + lane < c.ngc)
        s[c.gc_off + TILE * J + lane] = ((part[0][lane] + part[1][lane]) + part[2][lane]) + part[3][lane];
}

__global__ void __launch_bounds__(128) k_msym_reduce(const int2 *__restrict__ mt, const ClusterDev *__restrict__ cl,
                                                     const double *D, const double *P, double *s,
                                                     const PcpgState *st) {
    __shared__ double part[4][TILE];
    pdl_next();
    const int2 b = mt[blockIdx.x];
    const ClusterDev c = cl[b.x];
    const int J = b.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_wait();
    if (st && st->done) return;
    double y = warp == 0 ? D[((long long)c.mt_row_off + J) * TILE + lane] : 0.0;
#pragma unroll 4
    for (int I = J + 1 + warp; I < c.mt; I += 4) y += P[(c.MT_off + (long long)I * (I + 1) / 2 + J) * TILE + lane];
    part[warp][lane] = y;
    __syncthreads();
    if (warp == 0 && TILE * J + lane < c.ngc)
        s[c.gc_off + TILE * J + lane] = ((part[0][lane] + part[1][lane]) + part[2][lane]) + part[3][lane];
}

}  // namespace htf

// Gauge moves on the device: blocked Householder QR and its uses.
//
// The reference moves the orthogonality centre with the polar factor of an
// SVD (zgesdd, core.f95:2708-2960): A = (U S U^H)(U V^H).  Energies, overlaps
// and environments are invariant under any gauge A = P Q with Q having
// orthonormal rows, so the device path uses the Householder QR of A^H
// instead (A^H = Qt Rt, Q = Qt^H, P = Rt^H): it is backward stable for
// rank-deficient sites (Schmidt values down to zero), needs no iterative SVD
// and maps onto GEMMs.
//
// QR layout: right-looking blocked Householder, outer blocks of NB=64 columns
// (trailing update = three complex GEMMs through the compact WY form
// I - V T V^H).  Each block is factorised by one thread-block cluster of up
// to 16 CTAs with the block held in registers (mp <= 2048 rows); devices
// that cannot co-schedule such a cluster use inner panels of JB=4 columns
// (one CTA each) and a per-column update kernel.  Q is formed explicitly by
// backward accumulation of the block reflectors (zungqr order) or, in the
// look-ahead form, from the compact-WY factor of all of them.
#include <algorithm>
#include <cmath>
#include <memory>
#include <vector>

#include <cooperative_groups.h>

#include "nc_common.cuh"
#include "nc_kernels.h"

namespace nc {

namespace cg = cooperative_groups;

namespace {

constexpr int JB = 4;      // panel width
constexpr int NB = 64;     // outer block width
constexpr int PT = 256;    // panel threads
constexpr int PMAXROWS = 8;  // rows per thread -> mp <= 2048

template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double* red, double* out) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        double x = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) red[wid * NV + k] = x;
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        double s = 0;
        for (int w = 0; w < PT / 32; ++w) s += red[w * NV + threadIdx.x];
        out[threadIdx.x] = s;
    }
    __syncthreads();
}

// Factor the mp x jb panel at A (ld lda), jb <= JB.  Writes R (upper part)
// and the reflector tails back to A, the unit-diagonal reflectors to V
// (ld ldv, rows 0..mp-1), tau, and the JB x JB compact-WY T.
template <int ROWS>
__global__ void __launch_bounds__(PT) panel_qr_kernel(int mp, int jb, cplx* __restrict__ A, long long lda,
                                                      cplx* __restrict__ V, long long ldv,
                                                      cplx* __restrict__ tau_out, cplx* __restrict__ Tout) {
    __shared__ double red[(PT / 32) * 2 * JB * JB];
    __shared__ double outv[2 * JB * JB];
    __shared__ cplx s_alpha;
    __shared__ cplx s_tau[JB];
    const int tid = threadIdx.x;
    cplx a[ROWS][JB];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        int row = tid + r * PT;
#pragma unroll
        for (int c = 0; c < JB; ++c) a[r][c] = (row < mp && c < jb) ? A[row + c * lda] : cmake(0, 0);
    }
#pragma unroll
    for (int c = 0; c < JB; ++c) {  // unrolled so that a[][c] stays in registers
        if (c >= jb) break;
        double p[1] = {0.0};
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            int row = tid + r * PT;
            if (row > c && row < mp) p[0] += cabs2(a[r][c]);
            if (row == c) s_alpha = a[r][c];
        }
        block_sum<1>(p, red, outv);
        const double xnorm2 = outv[0];
        const cplx alpha = s_alpha;
        cplx t = cmake(0, 0), scale = cmake(1, 0), diag = alpha;
        if (!(xnorm2 == 0.0 && alpha.y == 0.0)) {
            double beta = -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xnorm2), alpha.x);
            t = cmake((beta - alpha.x) / beta, -alpha.y / beta);
            cplx den = cmake(alpha.x - beta, alpha.y);
            double dd = den.x * den.x + den.y * den.y;
            scale = cmake(den.x / dd, -den.y / dd);
            diag = cmake(beta, 0);
        }
        double w[2 * JB];
#pragma unroll
        for (int k = 0; k < 2 * JB; ++k) w[k] = 0;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            int row = tid + r * PT;
            cplx v = cmake(0, 0);
            if (row == c) { a[r][c] = diag; v = cmake(1, 0); }
            else if (row > c && row < mp) { a[r][c] = cmul(a[r][c], scale); v = a[r][c]; }
            cplx vc = cconj(v);
#pragma unroll
            for (int c2 = 0; c2 < JB; ++c2) {
                if (c2 > c) {
                    cplx q = cmul(vc, a[r][c2]);
                    w[2 * c2] += q.x;
                    w[2 * c2 + 1] += q.y;
                }
            }
        }
        block_sum<2 * JB>(w, red, outv);
        const cplx tc = cconj(t);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            int row = tid + r * PT;
            if (row < c || row >= mp) continue;
            cplx v = (row == c) ? cmake(1, 0) : a[r][c];
#pragma unroll
            for (int c2 = 0; c2 < JB; ++c2) {
                if (c2 > c && c2 < jb) {
                    cplx wc = cmake(outv[2 * c2], outv[2 * c2 + 1]);
                    a[r][c2] = csub(a[r][c2], cmul(tc, cmul(v, wc)));
                }
            }
        }
        if (tid == 0) s_tau[c] = t;
        __syncthreads();
    }
    // write back and Gram matrix of the reflectors
    double g[2 * JB * JB];
#pragma unroll
    for (int k = 0; k < 2 * JB * JB; ++k) g[k] = 0;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        int row = tid + r * PT;
        if (row >= mp) continue;
        cplx v[JB];
#pragma unroll
        for (int c = 0; c < JB; ++c) {
            v[c] = (c >= jb || row < c) ? cmake(0, 0) : (row == c ? cmake(1, 0) : a[r][c]);
            if (c < jb) {
                A[row + c * lda] = a[r][c];
                V[row + c * ldv] = v[c];
            }
        }
#pragma unroll
        for (int k = 0; k < JB; ++k)
#pragma unroll
            for (int c = 0; c < JB; ++c) {
                if (k < c) {
                    cplx q = cmul(cconj(v[k]), v[c]);
                    g[2 * (k + JB * c)] += q.x;
                    g[2 * (k + JB * c) + 1] += q.y;
                }
            }
    }
    block_sum<2 * JB * JB>(g, red, outv);
    if (tid == 0) {
        // compact WY (zlarft, forward/columnwise): T(c,c) = tau_c,
        // T(0:c,c) = -tau_c T(0:c,0:c) V(:,0:c)^H v_c
        cplx T[JB][JB];
        for (int i = 0; i < JB; ++i)
            for (int j = 0; j < JB; ++j) T[i][j] = cmake(0, 0);
        for (int c = 0; c < jb; ++c) {
            cplx tc = s_tau[c];
            T[c][c] = tc;
            for (int k = 0; k < c; ++k) {
                cplx acc = cmake(0, 0);
                for (int l = k; l < c; ++l)
                    acc = cadd(acc, cmul(T[k][l], cmake(outv[2 * (l + JB * c)], outv[2 * (l + JB * c) + 1])));
                T[k][c] = cscale(cmul(tc, acc), -1.0);
            }
        }
        for (int i = 0; i < JB; ++i)
            for (int j = 0; j < JB; ++j) Tout[i + JB * j] = T[i][j];
        for (int c = 0; c < jb; ++c) tau_out[c] = s_tau[c];
    }
}

// Apply the panel's (I - V T V^H)^H to nc columns of A (one block per column):
// a -= V T^H (V^H a).
__global__ void __launch_bounds__(PT) panel_apply_kernel(int mp, int jb, const cplx* __restrict__ V,
                                                         long long ldv, const cplx* __restrict__ T,
                                                         cplx* __restrict__ A, long long lda) {
    __shared__ double red[(PT / 32) * 2 * JB];
    __shared__ double outv[2 * JB];
    cplx* col = A + (long long)blockIdx.x * lda;
    double w[2 * JB];
#pragma unroll
    for (int k = 0; k < 2 * JB; ++k) w[k] = 0;
    for (int row = threadIdx.x; row < mp; row += PT) {
        cplx x = col[row];
#pragma unroll
        for (int c = 0; c < JB; ++c) {
            if (c < jb) {
                cplx q = cmul(cconj(V[row + c * ldv]), x);
                w[2 * c] += q.x;
                w[2 * c + 1] += q.y;
            }
        }
    }
    block_sum<2 * JB>(w, red, outv);
    // w2 = T^H w
    cplx w2[JB];
#pragma unroll
    for (int i = 0; i < JB; ++i) {
        cplx acc = cmake(0, 0);
        for (int k = 0; k <= i && k < jb; ++k)
            acc = cadd(acc, cmul(cconj(T[k + JB * i]), cmake(outv[2 * k], outv[2 * k + 1])));
        w2[i] = acc;
    }
    for (int row = threadIdx.x; row < mp; row += PT) {
        cplx x = col[row];
#pragma unroll
        for (int c = 0; c < JB; ++c)
            if (c < jb) x = csub(x, cmul(V[row + c * ldv], w2[c]));
        col[row] = x;
    }
}

// Compact-WY T (nb x nb, forward/columnwise: H_0 H_1 ... = I - V T V^H) from
// the strict upper part of G = V^H V and tau, by recursive doubling: with T
// known on two adjacent diagonal blocks a, b of size s,
//   T(a,b) = -T(a,a) G(a,b) T(b,b)
// (the block form of the zlarft recurrence; Puglisi 1992, Joffrain et al.
// 2006), so six levels of small block products build the 64 x 64 T.  One
// CTA, T, G and the level's products in shared memory.
constexpr int BT_T = 1024;
constexpr size_t BT_SMEM = sizeof(cplx) * ((size_t)2 * NB * (NB + 1) + NB * NB / 2);

// G: ld nb.
__global__ void __launch_bounds__(BT_T) build_t_kernel(int nb, const cplx* __restrict__ G, const cplx* __restrict__ tau, cplx* __restrict__ T,
                                                      int ldt) {
    extern __shared__ __align__(16) unsigned char bt_smem[];
    cplx* Ts = reinterpret_cast<cplx*>(bt_smem);   // [NB][NB+1]
    cplx* Gs = Ts + NB * (NB + 1);                   // [NB][NB+1], strict upper part
    cplx* Xs = Gs + NB * (NB + 1);                   // one level's G(a,b) T(b,b) blocks
    const int tid = threadIdx.x;
    for (int e = tid; e < NB * NB; e += BT_T) {
        const int i = e % NB, j = e / NB;
        cplx g = cmake(0, 0);
        if (i < j && j < nb) g = G[i + (long long)nb * j];
        Gs[i * (NB + 1) + j] = g;
        Ts[i * (NB + 1) + j] = (i == j && i < nb) ? tau[i] : cmake(0, 0);
    }
    __syncthreads();
    for (int s = 1; s < NB; s <<= 1) {
        const int per = s * s, total = (NB / (2 * s)) * per;
        for (int e = tid; e < total; e += BT_T) {   // X = G(a,b) T(b,b), T(b,b) upper
            const int pr = e / per, rem = e % per, i = rem / s, j = rem % s;
            const int a0 = 2 * pr * s, b0 = a0 + s;
            double xr = 0, xi = 0;
            for (int l = 0; l <= j; ++l) {
                const cplx g = Gs[(a0 + i) * (NB + 1) + b0 + l], t = Ts[(b0 + l) * (NB + 1) + b0 + j];
                xr = fma(g.x, t.x, fma(-g.y, t.y, xr));
                xi = fma(g.x, t.y, fma(g.y, t.x, xi));
            }
            Xs[e] = cmake(xr, xi);
        }
        __syncthreads();
        for (int e = tid; e < total; e += BT_T) {   // T(a,b) = -T(a,a) X, T(a,a) upper
            const int pr = e / per, rem = e % per, i = rem / s, j = rem % s;
            const int a0 = 2 * pr * s, b0 = a0 + s;
            double tr = 0, ti = 0;
            for (int l = i; l < s; ++l) {
                const cplx t = Ts[(a0 + i) * (NB + 1) + a0 + l], x = Xs[pr * per + l * s + j];
                tr = fma(t.x, x.x, fma(-t.y, x.y, tr));
                ti = fma(t.x, x.y, fma(t.y, x.x, ti));
            }
            Ts[(a0 + i) * (NB + 1) + b0 + j] = cmake(-tr, -ti);
        }
        __syncthreads();
    }
    for (int e = tid; e < NB * NB; e += BT_T) {
        const int i = e % NB, j = e / NB;
        T[i + (long long)ldt * j] = Ts[i * (NB + 1) + j];
    }
}

void launch_build_t(Context& ctx, int nb, const cplx* G, const cplx* tau, cplx* T) {
    NC_SET_SMEM_ONCE(build_t_kernel, BT_SMEM);
    build_t_kernel<<<1, BT_T, BT_SMEM, ctx.stream>>>(nb, G, tau, T, NB);
    NC_CHECK_LAUNCH();
    ctx.launches++;
}

// W2 = T^H W (nb x nc) without forming T: T^-H = diag(1 / conj(tau)) + the strict
// lower part of V^H V (the compact-WY identity T^-1 + T^-H = V^H V), so W2 comes
// out of a forward substitution, one warp per column and G = V^H V in shared
// memory.  64 dependent steps, 8 us on a B200, where building T takes 27 us and
// multiplying by it another 14.
constexpr int TRS_WARPS = 4;
constexpr size_t TRS_SMEM = sizeof(cplx) * NB * NB;
__global__ void __launch_bounds__(32 * TRS_WARPS) reflector_solve_kernel(int nb, int nc, const cplx* __restrict__ G,
                                                                         const cplx* __restrict__ tau,
                                                                         const cplx* __restrict__ W,
                                                                         cplx* __restrict__ W2) {
    extern __shared__ __align__(16) unsigned char trs_smem[];
    cplx* Gs = reinterpret_cast<cplx*>(trs_smem);   // column-major, ld nb
    __shared__ cplx ts[NB];
    for (int e = threadIdx.x; e < nb * nb; e += 32 * TRS_WARPS) Gs[e] = G[e];
    for (int e = threadIdx.x; e < nb; e += 32 * TRS_WARPS) ts[e] = cconj(tau[e]);
    __syncthreads();
    const int lane = threadIdx.x & 31, k = blockIdx.x * TRS_WARPS + (threadIdx.x >> 5);
    if (k >= nc) return;
    cplx w0 = lane < nb ? W[lane + (long long)nb * k] : cmake(0, 0);
    cplx w1 = lane + 32 < nb ? W[lane + 32 + (long long)nb * k] : cmake(0, 0);
    for (int i = 0; i < nb; ++i) {
        const cplx own = i < 32 ? w0 : w1;
        cplx v = cmake(__shfl_sync(0xffffffffu, own.x, i & 31), __shfl_sync(0xffffffffu, own.y, i & 31));
        v = cmul(ts[i], v);
        const cplx* g = Gs + i * nb;
        if (lane == i) w0 = v;
        else if (lane > i && lane < nb) w0 = csub(w0, cmul(g[lane], v));
        if (lane + 32 == i) w1 = v;
        else if (lane + 32 > i && lane + 32 < nb) w1 = csub(w1, cmul(g[lane + 32], v));
    }
    if (lane < nb) W2[lane + (long long)nb * k] = w0;
    if (lane + 32 < nb) W2[lane + 32 + (long long)nb * k] = w1;
}

// Zeros above the diagonal blocks of V (columns c, rows < NB floor(c / NB)) and
// in the whole of T (n x n).
__global__ void zero_upper_kernel(int n, cplx* __restrict__ V, long long ldv, cplx* __restrict__ T) {
    const long long total = (long long)n * n;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(e % n), c = (int)(e / n);
        T[e] = cmake(0, 0);
        if (r < c / NB * NB) V[r + c * ldv] = cmake(0, 0);
    }
}

// The nb x nb block T (ld NB) to the diagonal of the full factor (ld n).
__global__ void place_t_kernel(int nb, const cplx* __restrict__ T, cplx* __restrict__ full, long long ldf) {
    for (int e = threadIdx.x; e < nb * nb; e += blockDim.x) full[e % nb + (e / nb) * ldf] = T[e % nb + NB * (e / nb)];
}

// Q <- I - Q (m x n)
__global__ void one_minus_kernel(long long m, int n, cplx* __restrict__ Q) {
    const long long total = m * n;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const cplx q = Q[e];
        Q[e] = cmake((e % m == e / m ? 1.0 : 0.0) - q.x, -q.y);
    }
}

// ---------------------------------------------------------------------------
// One outer block (mp x nb, nb <= NB) factorised by a thread-block cluster.
//
// The rows are split over the C CTAs of one cluster (at most CQ_MAXR rows
// each, held in registers: thread (k, g) owns column k at rows g + 8i), so
// the whole block needs one launch instead of NB/JB panel and update
// launches.  Column j needs a single cluster-wide reduction: every CTA forms,
// over its rows below the diagonal,
//   s_k = sum_r conj(x_r) P(r,k)   for k >= j   (x = column j)
// which gives the column norm (k = j) and the reflector products with the
// trailing columns (k > j: w_k = P(j,k) + conj(scale) s_k), because
// v = e_j + scale * x; warps whose columns all lie left of j sit the column
// out (the Gram matrix V^H V of the compact-WY T is one GEMM after the
// kernel).  Each CTA stores its partial sums (and CTA 0,
// which holds the pivot rows, row j) into every CTA's shared memory (DSMEM,
// double-buffered by column parity) and one cluster barrier publishes them;
// each CTA then reduces the C partials with the same tree, so all CTAs
// derive bit-identical reflectors.  Reflector tails stay unscaled; the scale
// of column k is applied on use and at write-back.  The only waits are the
// hardware block and cluster barriers.
// ---------------------------------------------------------------------------
constexpr int CQ_T = 512;             // threads per CTA
constexpr int CQ_G = CQ_T / NB;       // lanes per column (row interleave)
constexpr int CQ_MAXC = 16;           // CTAs per cluster (non-portable size)
constexpr int CQ_MAXR = 128;          // rows per CTA -> mp <= 2048
constexpr int CQ_RPT = CQ_MAXR / CQ_G;  // rows per thread
__global__ void __launch_bounds__(CQ_T, 1)
cluster_block_qr_kernel(int mp, int nb, int rows_per_cta, cplx* __restrict__ A, long long lda,
                        cplx* __restrict__ V, long long ldv, cplx* __restrict__ tau_out) {
    __shared__ cplx recv[2][CQ_MAXC][NB];   // partial sums by source CTA, per column parity
    __shared__ cplx piv[2][NB];             // pivot row as received, per column parity
    __shared__ cplx pivst[2][NB];           // pivot row staged by its owners (CTA 0)
    __shared__ cplx xs[2][CQ_MAXR];         // column j of this CTA's rows
    __shared__ cplx colscale[NB];
    __shared__ cplx taus[NB];
    cg::cluster_group cluster = cg::this_cluster();
    const int C = (int)cluster.num_blocks();
    const int rank = (int)cluster.block_rank();
    const int tid = threadIdx.x, k = tid / CQ_G, g = tid % CQ_G;
    const int row0 = rank * rows_per_cta;
    const int nr = max(0, min(rows_per_cta, mp - row0));
    // Row j (< nb) always lies in CTA 0: rows_per_cta >= nb whenever C > 1
    // (mp > CQ_MAXR (C-1)), and mp >= nb when C == 1.
    const bool top = (rank == 0);

    cplx a[CQ_RPT];
#pragma unroll
    for (int i = 0; i < CQ_RPT; ++i) {
        const int r = g + CQ_G * i;
        a[i] = (r < nr && k < nb) ? A[(row0 + r) + (long long)k * lda] : cmake(0, 0);
    }
    if (k == 0) {
#pragma unroll
        for (int i = 0; i < CQ_RPT; ++i) xs[0][g + CQ_G * i] = a[i];
    }
    if (top && g == 0) pivst[0][k] = a[0];   // row 0
    cluster.sync();

    for (int j = 0; j < nb; ++j) {
        const int p = j & 1;
        // Only columns k >= j take part in column j; a warp whose four
        // columns all lie left of j (k = 4*warp .. 4*warp + 3) skips it.
        const bool wactive = 4 * (tid >> 5) + 3 >= j;
        if (wactive) {
            // phase 1: partial sums over this CTA's rows below the diagonal.
            // Only CTA 0's first NB rows can lie on or above the diagonal.
            double s0r = 0, s0i = 0, s1r = 0, s1i = 0;
#pragma unroll
            for (int i = 0; i < CQ_RPT; i += 2) {
                const int r0 = g + CQ_G * i, r1 = r0 + CQ_G;
                const cplx x0 = xs[p][r0], x1 = xs[p][r1];
                const bool u0 = !top || r0 >= NB || r0 > j, u1 = !top || r1 >= NB || r1 > j;
                if (u0) {
                    s0r = fma(x0.x, a[i].x, fma(x0.y, a[i].y, s0r));
                    s0i = fma(x0.x, a[i].y, fma(-x0.y, a[i].x, s0i));
                }
                if (u1) {
                    s1r = fma(x1.x, a[i + 1].x, fma(x1.y, a[i + 1].y, s1r));
                    s1i = fma(x1.x, a[i + 1].y, fma(-x1.y, a[i + 1].x, s1i));
                }
            }
            double sr = s0r + s1r, si = s0i + s1i;
#pragma unroll
            for (int o = 1; o < CQ_G; o <<= 1) {
                sr += __shfl_xor_sync(0xffffffffu, sr, o);
                si += __shfl_xor_sync(0xffffffffu, si, o);
            }
            // phase 2: push to every CTA of the cluster (DSMEM stores)
            if (k >= j) {
                const cplx part = cmake(sr, si);
                const cplx pv = top ? pivst[p][k] : cmake(0, 0);
                for (int d = g; d < C; d += CQ_G) {
                    cluster.map_shared_rank(&recv[p][rank][0], d)[k] = part;
                    if (top) cluster.map_shared_rank(&piv[p][0], d)[k] = pv;
                }
            }
        }
        cluster.sync();   // release/acquire: publishes the partial sums
        if (wactive) {
            // phase 3: the CQ_G lanes of column k split the sources; a fixed
            // reduction tree keeps every CTA bit-identical
            cplx Sk = cmake(0, 0), Sj = cmake(0, 0);
            for (int c = g; c < C; c += CQ_G) {
                Sk = cadd(Sk, recv[p][c][k]);
                Sj = cadd(Sj, recv[p][c][j]);
            }
#pragma unroll
            for (int o = 1; o < CQ_G; o <<= 1) {
                Sk.x += __shfl_xor_sync(0xffffffffu, Sk.x, o);
                Sk.y += __shfl_xor_sync(0xffffffffu, Sk.y, o);
                Sj.x += __shfl_xor_sync(0xffffffffu, Sj.x, o);
            }
            const double xnorm2 = Sj.x;
            const cplx alpha = piv[p][j];
            const cplx pk = piv[p][k];
            cplx t = cmake(0, 0), scale = cmake(1, 0), diag = alpha;
            const bool reflect = !(xnorm2 == 0.0 && alpha.y == 0.0);
            if (reflect) {
                const double beta = -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xnorm2), alpha.x);
                const cplx den = cmake(alpha.x - beta, alpha.y);
                const double ib = 1.0 / beta;
                const double idd = 1.0 / (den.x * den.x + den.y * den.y);
                t = cmake((beta - alpha.x) * ib, -alpha.y * ib);
                scale = cmake(den.x * idd, -den.y * idd);
                diag = cmake(beta, 0);
            }
            if (k == j && g == 0) {
                colscale[j] = scale;
                taus[j] = t;
            }
            // phase 4: apply H_j^H = I - conj(tau) v v^H to the trailing columns
            if (reflect && k > j && k < nb) {
                const cplx cf = cmul(cconj(t), cadd(pk, cmul(cconj(scale), Sk)));
                const cplx ef = cmul(scale, cf);
                if (top) {
#pragma unroll
                    for (int i = 0; i < CQ_RPT; ++i) {
                        const int r = g + CQ_G * i;
                        if (r < NB && r == j) a[i] = csub(a[i], cf);
                        else if (r >= NB || r > j) a[i] = csub(a[i], cmul(xs[p][r], ef));
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < CQ_RPT; ++i) a[i] = csub(a[i], cmul(xs[p][g + CQ_G * i], ef));
                }
            }
            if (top && k >= j) {
                // diagonal of R, and stage row j+1 for the next pivot broadcast
#pragma unroll
                for (int i = 0; i < CQ_RPT / 2; ++i) {   // rows < NB
                    const int r = g + CQ_G * i;
                    if (k == j && r == j) a[i] = diag;
                    if (r == j + 1) pivst[p ^ 1][k] = a[i];
                }
            }
            if (k == j + 1) {
#pragma unroll
                for (int i = 0; i < CQ_RPT; ++i) xs[p ^ 1][g + CQ_G * i] = a[i];
            }
        }
        __syncthreads();
    }

    {
#pragma unroll
        for (int i = 0; i < CQ_RPT; ++i) {
            const int r = g + CQ_G * i, prow = row0 + r;
            if (r < nr && k < nb) {
                cplx v = a[i];
                if (prow > k) v = cmul(v, colscale[k]);
                A[prow + (long long)k * lda] = v;
                V[prow + (long long)k * ldv] = (prow > k) ? v : cmake(prow == k ? 1.0 : 0.0, 0);
            }
        }
        if (rank == 0)
            for (int c = tid; c < nb; c += CQ_T) tau_out[c] = taus[c];
    }
    cluster.sync();   // no CTA leaves while another may still write its shared memory
}

// ---------------------------------------------------------------------------
// The same block factorised eight columns at a time, for the shapes of more
// than one block.
//
// What bounds cluster_block_qr_kernel is the chain of one column: partial sums
// of all trailing columns (FP64 pipe), exchange, reflector, update of all
// trailing columns (FP64 pipe), 3.3 us of it at 16 CTAs.  Here the chain of a
// column only involves the eight columns of its sub-block: thread (c, r) holds
// rows r and r + 64 of column c, two rows instead of sixteen.  The other
// columns get the eight reflectors at once,
//   P <- P - V W2,  W2 = T^H (V^H P)  (T 8 x 8, compact WY),
// on the FP64 tensor pipe (M = 8 reflectors or columns fits its m8n8k4 shape),
// with V^H P summed over the CTAs by column slices once per sub-block.  v_c^H v_i for i < c
// comes out of the column's own sums (they run over all eight columns), so it
// costs nothing.  B200, one 2048 x 64 block: 212 -> 174
// us, 166 in the mean of the sixteen blocks of a 2048 x 1024 QR.
//
// The one-block shapes (n <= 64) keep the kernel above: their results stay what
// they were bit for bit (a chain's edge sites turn rounding into the phase of
// the state).
// ---------------------------------------------------------------------------
constexpr int SB = 8;             // columns per sub-block
constexpr int VP = CQ_MAXR + 1;   // pitch of the reflectors: neighbours start in neighbouring banks
constexpr int RS = 640;           // C x ceil(64 / C) x SB at most, over C = 1 .. 16
struct SubSmem {
    cplx recvW[RS];                   // V^H P partial sums of this CTA's columns, by source CTA
    cplx recv[2][SB][2 * CQ_MAXC];    // column sums by source half CTA, per column parity
    cplx piv[2][SB];                  // pivot row, per column parity
    cplx xs[2][CQ_MAXR];              // the column's rows, per parity
    cplx v[SB][VP];                   // the reflectors, explicit
    cplx col[SB][CQ_MAXR];            // the columns: R above, beta on and v below the diagonal
    cplx part[NB][SB];                // V^H P over the second 64 rows; then W2
    cplx G[SB][SB];                   // G[c][i] = v_c^H v_i, i < c
    cplx T[SB][SB];                   // compact-WY factor of the sub-block, T[g][i] = conj(T(i, g))
    cplx tau[SB];
    cplx taus[NB];
    unsigned long long bar[2];        // arrival of a column's sums, per parity
};

// Remote stores whose arrival the receiver waits for on its own mbarrier
// (st.async): a column needs one way through the cluster, not a cluster barrier
// with its stores before it (2.9 -> 1.9 thousand cycles a column at 16 CTAs).
// The wait is bounded by the global timer and reports through the context's watch.
__device__ __forceinline__ uint32_t remote(const void* p, int cta) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(cta));
    return r;
}
__device__ __forceinline__ void send8(uint32_t to, double v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(to),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ bool arrived(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void wait_sums(uint32_t bar, uint32_t parity, bool& alive, const DeviceWatch* watch) {
    if (!alive || arrived(bar, parity)) return;
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    while (!arrived(bar, parity)) {
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        if (watch_over(watch, t1 - t0)) {   // give up for good: every later wait returns at once
            watch_expired(watch, WATCH_QR);
            alive = false;
            return;
        }
    }
}

__device__ __forceinline__ void qr_dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// Column g of the sub-block's T by one warp, lane i < SB:
// T(i,g) = -tau_g sum_{i<=l<g} T(i,l) v_l^H v_g, products first, then a tree.
__device__ __forceinline__ void t_column(SubSmem& s, int g, int lane) {
    if (lane >= SB) return;
    cplx x[SB];
#pragma unroll
    for (int l = 0; l < SB - 1; ++l) x[l] = l < g ? cmul(s.T[l][lane], s.G[g][l]) : cmake(0, 0);   // conjugates of both
    const cplx sum = cadd(cadd(cadd(x[0], x[1]), cadd(x[2], x[3])), cadd(cadd(x[4], x[5]), x[6]));
    const cplx tg = cconj(s.tau[g]);
    s.T[g][lane] = lane < g ? cscale(cmul(tg, sum), -1.0) : lane == g ? tg : cmake(0, 0);
}

__global__ void __launch_bounds__(CQ_T, 1)
cluster_subblock_qr_kernel(int mp, int nb, int rows_per_cta, cplx* __restrict__ A, long long lda,
                           cplx* __restrict__ V, long long ldv, cplx* __restrict__ tau_out,
                           const DeviceWatch* __restrict__ watch) {
    extern __shared__ __align__(16) unsigned char sub_smem[];
    SubSmem& s = *reinterpret_cast<SubSmem*>(sub_smem);
    cg::cluster_group cluster = cg::this_cluster();
    const int C = (int)cluster.num_blocks();
    const int rank = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31;
    // Whole block: warp (ct, h) holds columns 8 ct .. + 7, rows 64 h .. + 63; lane (n, q) column
    // 8 ct + n, rows 64 h + 8 t + 2 q + e in a[2 t + e].  That is the B operand of an m8n8k4 FP64
    // MMA with K over four of the rows (V^H P) and the accumulator of one with the columns as
    // its rows (P^T - W2^T V^T), so both run from registers.
    const int ct = tid >> 6, h = (tid >> 5) & 1, n = lane >> 2, q4 = lane & 3;
    const int k = 8 * ct + n, rbase = 64 * h + 2 * q4;
    const int c = tid >> 6, r0 = tid & 63, r1 = r0 + 64;       // sub-block: column c, rows r0 and r1
    const int row0 = rank * rows_per_cta;
    const int nr = max(0, min(rows_per_cta, mp - row0));
    const bool top = rank == 0;   // holds all pivot rows (rows_per_cta >= 64 whenever C > 1)
    int span = 2;                 // lanes that hold one column sum's sources: 2 C, rounded up to a power of two
    while (span < 2 * C) span <<= 1;
    const int slice = (NB + C - 1) / C;   // columns per CTA of the exchanged V^H P
    const uint32_t bars = (uint32_t)__cvta_generic_to_shared(s.bar);
    const uint32_t column_bytes = (uint32_t)C * SB * 2 * 16 + SB * 16;   // sums of C CTAs, the pivot row
    bool alive = true;   // this thread has not given up a wait
    const bool mute = rank == C - 1 && (watch->mute >> WATCH_QR & 1u);   // test switch: no sums for column 0
    if (tid == 0) {
        for (int b = 0; b < 2; ++b) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bars + 8 * b) : "memory");
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bars + 8 * b), "r"(column_bytes)
                         : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    static_assert(CQ_T == 64 * SB && CQ_MAXR == 128 && NB == 64, "thread layouts");

    cplx a[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int r = rbase + 8 * (i >> 1) + (i & 1);
        a[i] = (r < nr && k < nb) ? A[(row0 + r) + (long long)k * lda] : cmake(0, 0);
    }
    for (int c0 = 0; c0 < nb; c0 += SB) {
        const int w = min(SB, nb - c0);
        const bool owner = 8 * ct == c0;
        if (owner) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int r = rbase + 8 * (i >> 1) + (i & 1);
                s.col[n][r] = a[i];
                if (n == 0) s.xs[0][r] = a[i];
            }
        }
        if (c0 == 0) cluster.sync();   // every CTA runs before the first remote store
        else __syncthreads();
        cplx p0 = s.col[c][r0], p1 = s.col[c][r1];
        for (int jj = 0; jj < w; ++jj) {
            const int j = c0 + jj, p = jj & 1;
            // sums below the diagonal of conj(x) times every column of the sub-block
            const cplx x0 = s.xs[p][r0], x1 = s.xs[p][r1];
            double sr = 0, si = 0;
            if (!top || r0 > j) {
                sr = fma(x0.x, p0.x, x0.y * p0.y);
                si = fma(x0.x, p0.y, -x0.y * p0.x);
            }
            sr = fma(x1.x, p1.x, fma(x1.y, p1.y, sr));   // r1 >= 64 > j
            si = fma(x1.x, p1.y, fma(-x1.y, p1.x, si));
            {
                // lanes 0-15 go on with the real part, 16-31 with the imaginary one
                const bool up = lane & 16;
                const double pvx = __shfl_sync(0xffffffffu, p0.x, j & 31), pvy = __shfl_sync(0xffffffffu, p0.y, j & 31);
                const double pv = up ? pvy : pvx;   // the pivot row, in the warps that hold it
                double sum = (up ? si : sr) + __shfl_xor_sync(0xffffffffu, up ? sr : si, 16);
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                // lane d (and d + 16) to CTA d
                const int d = lane & 15;
                if (d < C && !(mute && j == 0)) {
                    const uint32_t bar = remote(&s.bar[p], d);
                    send8(remote(&s.recv[p][c][2 * rank + h], d) + (up ? 8 : 0), sum, bar);
                    if (top && h == (j >> 5)) send8(remote(&s.piv[p][c], d) + (up ? 8 : 0), pv, bar);
                }
            }
            if (tid < 32 && jj > 0) t_column(s, jj - 1, lane);   // while the sums travel
            wait_sums(bars + 8 * p, (uint32_t)(j >> 1) & 1u, alive, watch);
            // every thread: the totals of its column and of column jj, in a fixed tree
            const int src = lane & (span - 1);
            cplx Sc = src < 2 * C ? s.recv[p][c][src] : cmake(0, 0);
            double Sj = src < 2 * C ? s.recv[p][jj][src].x : 0.0;
            for (int o = span >> 1; o > 0; o >>= 1) {
                Sc.x += __shfl_xor_sync(0xffffffffu, Sc.x, o);
                Sc.y += __shfl_xor_sync(0xffffffffu, Sc.y, o);
                Sj += __shfl_xor_sync(0xffffffffu, Sj, o);
            }
            const cplx alpha = s.piv[p][jj], pc = s.piv[p][c];
            cplx t = cmake(0, 0), scale = cmake(1, 0), diag = alpha;
            const bool reflect = !(Sj == 0.0 && alpha.y == 0.0);
            if (reflect) {
                const double beta = -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + Sj), alpha.x);
                const cplx den = cmake(alpha.x - beta, alpha.y);
                const double ib = 1.0 / beta;
                const double idd = 1.0 / (den.x * den.x + den.y * den.y);
                t = cmake((beta - alpha.x) * ib, -alpha.y * ib);
                scale = cmake(den.x * idd, -den.y * idd);
                diag = cmake(beta, 0);
            }
            const bool below0 = !top || r0 > j;
            const cplx v0 = cmul(x0, scale), v1 = cmul(x1, scale);   // the reflector below its pivot
            if (c > jj) {
                if (reflect) {
                    const cplx cf = cmul(cconj(t), cadd(pc, cmul(cconj(scale), Sc)));
                    if (below0) p0 = csub(p0, cmul(v0, cf));
                    else if (r0 == j) p0 = csub(p0, cf);
                    p1 = csub(p1, cmul(v1, cf));
                }
                if (c == jj + 1) {
                    s.xs[p ^ 1][r0] = p0;
                    s.xs[p ^ 1][r1] = p1;
                }
            } else if (c == jj) {
                s.v[jj][r0] = below0 ? v0 : cmake(r0 == j ? 1.0 : 0.0, 0.0);
                s.v[jj][r1] = v1;
                if (below0) p0 = v0;
                else if (r0 == j) p0 = diag;
                p1 = v1;
                if (r0 == 0) {
                    s.tau[jj] = t;
                    s.taus[j] = t;
                }
            } else if (r0 == 0) {
                s.G[jj][c] = cadd(pc, cmul(cconj(scale), Sc));   // v_jj^H v_c, column c holding v_c below its pivot
            }
            __syncthreads();
            // every thread is past its wait: the barrier's next use is armed.  A thread that gave up does not
            // arm it (its phase has not ended) but goes on: the cluster's barriers count every thread
            if (tid == 0 && alive)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bars + 8 * p), "r"(column_bytes)
                             : "memory");
        }
        // the finished columns back to their owners: R above, beta on and v below the diagonal
        s.col[c][r0] = p0;
        s.col[c][r1] = p1;
        __syncthreads();
        if (owner && n < w) {
#pragma unroll
            for (int i = 0; i < 16; ++i) a[i] = s.col[n][rbase + 8 * (i >> 1) + (i & 1)];
        }
        if (c0 + SB >= nb) break;
        const bool mine = 8 * ct > c0;   // the warp's columns are to the right of the sub-block
        double wr[2] = {0, 0}, wi[2] = {0, 0};   // (V^H P)(lane / 4, 8 ct + 2 (lane % 4) + {0, 1})
        if (mine) {
            // four short chains of eight products (32 rows) each: half the rounding of one long chain
            double ur[4][2] = {}, ui[4][2] = {};
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const cplx v = s.v[n][rbase + 8 * (i >> 1) + (i & 1)];   // reflector n, this lane's row
                const int c2 = 2 * (i & 1);
                qr_dmma(ur[c2], v.x, a[i].x);
                qr_dmma(ur[c2 + 1], v.y, a[i].y);
                qr_dmma(ui[c2], v.x, a[i].y);
                qr_dmma(ui[c2 + 1], -v.y, a[i].x);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                wr[e] = (ur[0][e] + ur[1][e]) + (ur[2][e] + ur[3][e]);
                wi[e] = (ui[0][e] + ui[1][e]) + (ui[2][e] + ui[3][e]);
            }
            if (h == 1) {
                s.part[8 * ct + 2 * q4][n] = cmake(wr[0], wi[0]);
                s.part[8 * ct + 2 * q4 + 1][n] = cmake(wr[1], wi[1]);
            }
        } else if (tid < 32) {
            t_column(s, SB - 1, lane);   // warp 0 never holds columns to the right
        }
        __syncthreads();
        if (mine && h == 0) {
            // each column's sums go to the CTA that finishes it
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int kk = 8 * ct + 2 * q4 + e;
                const cplx u = s.part[kk][n];
                cluster.map_shared_rank(s.recvW, kk / slice)[(rank * slice + kk % slice) * SB + n] =
                    cmake(wr[e] + u.x, wi[e] + u.y);
            }
        }
        cluster.sync();
        {
            // W2 = T^H W, one column per eight lanes, sent to every CTA
            const int g = tid & 7, first = rank * slice, kk = first + (tid >> 3);
            const bool on = kk < min(NB, first + slice) && kk >= c0 + SB;
            cplx W = cmake(0, 0);
            if (on)
                for (int d = 0; d < C; ++d) W = cadd(W, s.recvW[(d * slice + kk - first) * SB + g]);
            cplx x[SB];
#pragma unroll
            for (int i = 0; i < SB; ++i) {
                x[i] = cmake(__shfl_sync(0xffffffffu, W.x, (lane & ~7) | i),
                             __shfl_sync(0xffffffffu, W.y, (lane & ~7) | i));
                x[i] = cmul(s.T[g][i], x[i]);   // zero for i > g
            }
            const cplx w2 = cadd(cadd(cadd(x[0], x[1]), cadd(x[2], x[3])), cadd(cadd(x[4], x[5]), cadd(x[6], x[7])));
            if (on)
                for (int d = 0; d < C; ++d) cluster.map_shared_rank(&s.part[kk][0], d)[g] = w2;
        }
        cluster.sync();
        if (mine) {
            const cplx w0 = s.part[k][q4], w1 = s.part[k][q4 + 4];
#pragma unroll
            for (int t8 = 0; t8 < 8; ++t8) {
                double cr[2] = {0, 0}, ci[2] = {0, 0};   // V W2, taken from P once: one rounding at P's size
                const cplx v0 = s.v[q4][64 * h + 8 * t8 + n], v1 = s.v[q4 + 4][64 * h + 8 * t8 + n];
                qr_dmma(cr, w0.x, v0.x);
                qr_dmma(ci, w0.y, v0.x);
                qr_dmma(cr, -w0.y, v0.y);
                qr_dmma(ci, w0.x, v0.y);
                qr_dmma(cr, w1.x, v1.x);
                qr_dmma(ci, w1.y, v1.x);
                qr_dmma(cr, -w1.y, v1.y);
                qr_dmma(ci, w1.x, v1.y);
                a[2 * t8] = csub(a[2 * t8], cmake(cr[0], ci[0]));
                a[2 * t8 + 1] = csub(a[2 * t8 + 1], cmake(cr[1], ci[1]));
            }
        }
        __syncthreads();   // s.v, s.col, s.part are rewritten by the next sub-block
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int r = rbase + 8 * (i >> 1) + (i & 1), prow = row0 + r;
        if (r < nr && k < nb) {
            A[prow + (long long)k * lda] = a[i];
            V[prow + (long long)k * ldv] = (prow > k) ? a[i] : cmake(prow == k ? 1.0 : 0.0, 0);
        }
    }
    if (top)
        for (int q = tid; q < nb; q += CQ_T) tau_out[q] = s.taus[q];
    cluster.sync();   // no CTA leaves while another may still write its shared memory
    if (!alive) {   // sums that nothing waited for may still be on their way: all are sent, 0.1 ms is ample
        unsigned long long t0, t1;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
        do asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        while (t1 - t0 < 100000ull);
    }
}

// Cluster launch support (size CQ_MAXC needs the non-portable opt-in); a
// device that cannot co-schedule the cluster uses the per-panel path.
// The attribute and the answer belong to each device, so both are kept per
// device (the first 64; others are probed on every call).
bool cluster_qr_probe() {
    if (cudaFuncSetAttribute(cluster_block_qr_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
            cudaSuccess ||
        cudaFuncSetAttribute(cluster_subblock_qr_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
            cudaSuccess ||
        cudaFuncSetAttribute(cluster_subblock_qr_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(SubSmem)) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CQ_MAXC);
    cfg.blockDim = dim3(CQ_T);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CQ_MAXC;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int nclusters = 0, nsub = 0;
    if (cudaOccupancyMaxActiveClusters(&nclusters, cluster_block_qr_kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    cfg.dynamicSmemBytes = sizeof(SubSmem);
    if (cudaOccupancyMaxActiveClusters(&nsub, cluster_subblock_qr_kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return nclusters >= 1 && nsub >= 1;
}

bool cluster_qr_available() {
    static std::atomic<int> state[64];   // 0 unknown, 1 available, 2 not available
    int dev = 0;
    NC_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return cluster_qr_probe();
    int s = state[dev].load(std::memory_order_acquire);
    if (s == 0) {
        s = cluster_qr_probe() ? 1 : 2;
        state[dev].store(s, std::memory_order_release);
    }
    return s == 1;
}

// `sub`: eight columns at a time (the shapes of several blocks).
void launch_cluster_block(Context& ctx, bool sub, int mp, int nb, cplx* A, long long lda, cplx* V, long long ldv,
                          cplx* tau) {
    const int C = std::max(1, std::min(CQ_MAXC, (mp + CQ_MAXR - 1) / CQ_MAXR));
    const int rows = (mp + C - 1) / C;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(CQ_T);
    cfg.stream = ctx.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (sub) {
        cfg.dynamicSmemBytes = sizeof(SubSmem);
        NC_CUDA(cudaLaunchKernelEx(&cfg, cluster_subblock_qr_kernel, mp, nb, rows, A, lda, V, ldv, tau,
                                   static_cast<const DeviceWatch*>(ctx.watch)));
    } else {
        NC_CUDA(cudaLaunchKernelEx(&cfg, cluster_block_qr_kernel, mp, nb, rows, A, lda, V, ldv, tau));
    }
    ctx.launches++;
}

__global__ void identity_cols(long long m, int n, cplx* __restrict__ Q) {
    const long long total = m * n;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        long long r = e % m, c = e / m;
        Q[e] = (r == c) ? cmake(1, 0) : cmake(0, 0);
    }
}

// R (n x n, zeros below) from the upper triangle of A (ld lda), optionally conjugated.
__global__ void extract_r(int n, const cplx* __restrict__ A, long long lda, bool conj, cplx* __restrict__ R) {
    const long long total = (long long)n * n;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        int r = (int)(e % n), c = (int)(e / n);
        cplx v = (r <= c) ? A[r + c * lda] : cmake(0, 0);
        R[e] = conj ? cconj(v) : v;
    }
}

unsigned gsz(long long n) {
    return (unsigned)std::max<long long>(1, std::min<long long>((n + 255) / 256, 148 * 16));
}

void launch_panel(Context& ctx, int mp, int jb, cplx* A, long long lda, cplx* V, long long ldv, cplx* tau,
                  cplx* T) {
    const int rows = (mp + PT - 1) / PT;
    if (rows <= 1) panel_qr_kernel<1><<<1, PT, 0, ctx.stream>>>(mp, jb, A, lda, V, ldv, tau, T);
    else if (rows <= 2) panel_qr_kernel<2><<<1, PT, 0, ctx.stream>>>(mp, jb, A, lda, V, ldv, tau, T);
    else if (rows <= 4) panel_qr_kernel<4><<<1, PT, 0, ctx.stream>>>(mp, jb, A, lda, V, ldv, tau, T);
    else panel_qr_kernel<8><<<1, PT, 0, ctx.stream>>>(mp, jb, A, lda, V, ldv, tau, T);
    NC_CHECK_LAUNCH();
    ctx.launches++;
}

}  // namespace

void householder_qr(Context& ctx, int m, int n, cplx* A, cplx* Q, cplx* R, bool conjR) {
    NC_ARG(m >= n && n >= 1, "householder_qr: need m >= n >= 1");
    NC_ARG(m <= PT * PMAXROWS, "householder_qr: at most 2048 rows (bond x physical dimension)");
    Arena& ar = ctx.scratch();
    ArenaFrame f(ar);
    const long long lda = m;
    cplx* V = ar.alloc_n<cplx>((size_t)m * n);
    cplx* tau = ar.alloc_n<cplx>(n);
    const int nblocks = (n + NB - 1) / NB;
    cplx* Tb = ar.alloc_n<cplx>((size_t)nblocks * NB * NB);
    cplx* T4 = ar.alloc_n<cplx>(JB * JB);
    cplx* G = ar.alloc_n<cplx>(NB * NB);
    cplx* W = ar.alloc_n<cplx>((size_t)NB * n);
    cplx* W2 = ar.alloc_n<cplx>((size_t)NB * n);
    const bool use_cluster = cluster_qr_available();
    if (!use_cluster) zfill(ctx, (long long)m * n, cmake(0, 0), V);
    for (int ob = 0; ob < nblocks; ++ob) {
        const int j0 = ob * NB;
        const int nb = std::min(NB, n - j0);
        const int mp = m - j0;
        const cplx* Vb = V + j0 + j0 * (long long)m;
        cplx* T = Tb + (size_t)ob * NB * NB;
        if (use_cluster) {
            launch_cluster_block(ctx, n > NB, mp, nb, A + j0 + j0 * lda, lda, V + j0 + j0 * (long long)m, m, tau + j0);
            zgemm(zgemm_params(OP_C, OP_N, nb, nb, mp, Vb, m, Vb, m, G, nb), ctx);
        } else {
            for (int jj = j0; jj < j0 + nb; jj += JB) {
                const int jb = std::min(JB, j0 + nb - jj);
                launch_panel(ctx, m - jj, jb, A + jj + jj * lda, lda, V + jj + jj * (long long)m, m, tau + jj,
                             T4);
                const int rest = j0 + nb - (jj + jb);
                if (rest > 0) {
                    panel_apply_kernel<<<rest, PT, 0, ctx.stream>>>(m - jj, jb, V + jj + jj * (long long)m, m,
                                                                    T4, A + jj + (jj + jb) * lda, lda);
                    NC_CHECK_LAUNCH();
                    ctx.launches++;
                }
            }
            zgemm(zgemm_params(OP_C, OP_N, nb, nb, mp, Vb, m, Vb, m, G, nb), ctx);
        }
        // compact WY T for the outer block from G = V^H V (strict upper part)
        launch_build_t(ctx, nb, G, tau + j0, T);
        // trailing update: A2 -= V T^H (V^H A2)
        const int nt = n - (j0 + nb);
        if (nt > 0) {
            cplx* A2 = A + j0 + (j0 + nb) * lda;
            zgemm(zgemm_params(OP_C, OP_N, nb, nt, mp, Vb, m, A2, lda, W, nb), ctx);
            zgemm(zgemm_params(OP_C, OP_N, nb, nt, nb, T, NB, W, nb, W2, nb), ctx);
            ZGemmParams p = zgemm_params(OP_N, OP_N, mp, nt, nb, Vb, m, W2, nb, A2, lda);
            p.alpha = cmake(-1, 0);
            p.beta = cmake(1, 0);
            zgemm(p, ctx);
        }
    }
    if (R) {
        extract_r<<<gsz((long long)n * n), 256, 0, ctx.stream>>>(n, A, lda, conjR, R);
        NC_CHECK_LAUNCH();
        ctx.launches++;
    }
    if (Q) {
        identity_cols<<<gsz((long long)m * n), 256, 0, ctx.stream>>>(m, n, Q);
        NC_CHECK_LAUNCH();
        ctx.launches++;
        for (int ob = nblocks - 1; ob >= 0; --ob) {
            const int j0 = ob * NB;
            const int nb = std::min(NB, n - j0);
            const int mp = m - j0;
            const int nq = n - j0;
            const cplx* Vb = V + j0 + j0 * (long long)m;
            const cplx* T = Tb + (size_t)ob * NB * NB;
            cplx* Qs = Q + j0 + j0 * (long long)m;
            // Qs = (I - V T V^H) Qs
            zgemm(zgemm_params(OP_C, OP_N, nb, nq, mp, Vb, m, Qs, m, W, nb), ctx);
            zgemm(zgemm_params(OP_N, OP_N, nb, nq, nb, T, NB, W, nb, W2, nb), ctx);
            ZGemmParams p = zgemm_params(OP_N, OP_N, mp, nq, nb, Vb, m, W2, nb, Qs, m);
            p.alpha = cmake(-1, 0);
            p.beta = cmake(1, 0);
            zgemm(p, ctx);
        }
    }
}

// Look-ahead form of householder_qr for the gauge moves (cluster path only).
// The main stream (ctx) runs the critical path: factor block k, then apply its
// reflector to block k+1 only, so that block k+1 can be factorised next: one
// batched product [V^H V, V^H A_{k+1}], a forward substitution in place of T
// (reflector_solve_kernel) and one rank-64 update.  Beside it the second stream
// builds T_k, applies the reflector to the remaining columns and extends the
// compact-WY factor of all reflectors so far,
//   T <- [T, -T (V^H V_k) T_k; 0, T_k],
// so that Q needs no pass per block: once the last block is done,
// Q(:, :n) = I - V (T V_1^H) (V_1 the top n rows of V) is two large products,
// through residues where those pay.
// On a B200 a chi = 1024 move (2048 x 1024) goes from 6.23 to 4.05 ms (with the
// panels of cluster_subblock_qr_kernel): per block the products between the
// panels took 130 us on the main stream (partial sums of V^H V and V^H A, T, W2,
// update), and accumulating Q forwards block by block kept the second stream
// busy for longer than the panels.
// ev: 2 + 2*nblocks events (fork, join, then per block: G ready, bulk update
// done).
// The dot products over the rows (V^H V, V^H A) are summed in chains of kDotChain
// rows and the chains added: one chain over all rows cost a third more error
// than the columns one at a time.  260 x 125, mean of 8 seeds, extended
// precision, columns one at a time / one chain / now: |Q^H Q - I| 1.09e-14 /
// 1.36e-14 / 9.2e-15, |A - QR| / |A| 8.2e-16 / 1.04e-15 / 7.4e-16,
// |R^H R - A^H A| / |A|^2 5.8e-17 / 9.5e-17 / 6.5e-17.
constexpr int kDotChain = 32;
// V (m x n, the reflectors) and T (n x n) are what qr_form_q takes.
void householder_qr_lookahead(Context& ctx, Context& side, cudaEvent_t* ev, int m, int n, cplx* A, cplx* V, cplx* T,
                              cplx* R, bool conjR) {
    NC_ARG(m >= n && n >= 1 && m <= CQ_MAXC * CQ_MAXR, "householder_qr: need 1 <= n <= m <= 2048");
    Arena& ar = ctx.scratch();
    ArenaFrame f(ar);
    const long long lda = m;
    const int nblocks = (n + NB - 1) / NB;
    cplx* tau = ar.alloc_n<cplx>(n);
    cplx* GW = ar.alloc_n<cplx>((size_t)nblocks * 2 * NB * NB);   // per block: V^H V, V^H A_{k+1}
    cplx* W2m = ar.alloc_n<cplx>(NB * NB);
    cplx* Tb = ar.alloc_n<cplx>(NB * NB);
    cplx* Ws = ar.alloc_n<cplx>((size_t)NB * n);
    cplx* W2s = ar.alloc_n<cplx>((size_t)NB * n);
    const uint64_t side0 = side.launches;
    NC_SET_SMEM_ONCE(reflector_solve_kernel, TRS_SMEM);

    NC_CUDA(cudaEventRecord(ev[0], ctx.stream));   // fork
    NC_CUDA(cudaStreamWaitEvent(side.stream, ev[0], 0));
    zero_upper_kernel<<<gsz((long long)n * n), 256, 0, side.stream>>>(n, V, m, T);
    NC_CHECK_LAUNCH();
    side.launches++;
    for (int ob = 0; ob < nblocks; ++ob) {
        const int j0 = ob * NB, nb = std::min(NB, n - j0), mp = m - j0;
        const int j1 = j0 + nb, nb1 = (ob + 1 < nblocks) ? std::min(NB, n - j1) : 0;
        const cplx* Vb = V + j0 + j0 * (long long)m;
        cplx* G = GW + (size_t)ob * 2 * NB * NB;
        cplx* W = G + NB * NB;
        cplx* A1 = A + j0 + j1 * lda;
        cudaEvent_t ev_g = ev[2 + 2 * ob], ev_bulk = ev[3 + 2 * ob];
        // main: factor block ob; its reflector on block ob+1, after the second
        // stream's update of those columns by reflector ob-1
        launch_cluster_block(ctx, true, mp, nb, A + j0 + j0 * lda, lda, V + j0 + j0 * (long long)m, m, tau + j0);
        if (nb1 > 0 && ob > 0) NC_CUDA(cudaStreamWaitEvent(ctx.stream, ev[3 + 2 * (ob - 1)], 0));
        ZGemmParams g = zgemm_params(OP_C, OP_N, nb, nb, mp, Vb, m, Vb, m, G, nb);
        g.chain = kDotChain;
        if (nb1 == nb) {   // both products as one batch: A and V have the same leading dimension
            g.batch = 2;
            g.sB0 = A1 - Vb;
            g.sC0 = NB * NB;
        }
        zgemm(g, ctx);
        if (nb1 > 0 && nb1 != nb) {
            ZGemmParams w = zgemm_params(OP_C, OP_N, nb, nb1, mp, Vb, m, A1, lda, W, nb);
            w.chain = kDotChain;
            zgemm(w, ctx);
        }
        NC_CUDA(cudaEventRecord(ev_g, ctx.stream));
        if (nb1 > 0) {
            reflector_solve_kernel<<<ceil_div(nb1, TRS_WARPS), 32 * TRS_WARPS, TRS_SMEM, ctx.stream>>>(nb, nb1, G, tau + j0,
                                                                                                      W, W2m);
            NC_CHECK_LAUNCH();
            ctx.launches++;
            ZGemmParams u = zgemm_params(OP_N, OP_N, mp, nb1, nb, Vb, m, W2m, nb, A1, lda);
            u.alpha = cmake(-1, 0);
            u.beta = cmake(1, 0);
            zgemm(u, ctx);
        }
        // side: T_ob, the reflector on the columns after block ob+1, the full T
        NC_CUDA(cudaStreamWaitEvent(side.stream, ev_g, 0));
        launch_build_t(side, nb, G, tau + j0, Tb);
        const int jr = j1 + nb1, nt = n - jr;
        if (nt > 0) {
            cplx* A2 = A + j0 + jr * lda;
            ZGemmParams w = zgemm_params(OP_C, OP_N, nb, nt, mp, Vb, m, A2, lda, Ws, nb);
            w.chain = kDotChain;
            zgemm(w, side);
            zgemm(zgemm_params(OP_C, OP_N, nb, nt, nb, Tb, NB, Ws, nb, W2s, nb), side);
            ZGemmParams p = zgemm_params(OP_N, OP_N, mp, nt, nb, Vb, m, W2s, nb, A2, lda);
            p.alpha = cmake(-1, 0);
            p.beta = cmake(1, 0);
            zgemm(p, side);
        }
        NC_CUDA(cudaEventRecord(ev_bulk, side.stream));
        place_t_kernel<<<1, 256, 0, side.stream>>>(nb, Tb, T + j0 + j0 * (long long)n, n);
        NC_CHECK_LAUNCH();
        side.launches++;
        if (j0 > 0) {
            // V(:, :j0)^H V_ob over the rows where V_ob is not zero
            ZGemmParams w = zgemm_params(OP_C, OP_N, j0, nb, mp, V + j0, m, Vb, m, Ws, j0);
            w.chain = kDotChain;
            zgemm(w, side);
            zgemm(zgemm_params(OP_N, OP_N, j0, nb, j0, T, n, Ws, j0, W2s, j0), side);
            ZGemmParams p = zgemm_params(OP_N, OP_N, j0, nb, nb, W2s, j0, Tb, NB, T + j0 * (long long)n, n);
            p.alpha = cmake(-1, 0);
            zgemm(p, side);
        }
    }
    NC_CUDA(cudaEventRecord(ev[1], side.stream));   // join
    NC_CUDA(cudaStreamWaitEvent(ctx.stream, ev[1], 0));
    ctx.launches += side.launches - side0;
    if (R) {
        extract_r<<<gsz((long long)n * n), 256, 0, ctx.stream>>>(n, A, lda, conjR, R);
        NC_CHECK_LAUNCH();
        ctx.launches++;
    }
}

// Q (m x n) = I - V (T V_1^H).  The reflectors and T are the QR's own, with
// errors of 2^-53 of their rows' norms, so the products are norm-wise: a bond with
// weights far apart gives V and T such rows too, and in FP64 the two products
// take 0.85 ms of a chi = 1024 move instead of 0.4.
void qr_form_q(Context& ctx, int m, int n, const cplx* V, const cplx* T, cplx* Q) {
    ArenaFrame f(ctx.scratch());
    cplx* Z = ctx.scratch().alloc_n<cplx>((size_t)n * n);
    ResMatrix a, b;
    a.X = T; a.rows = n; a.K = n; a.si = 1; a.sk = n; a.I = n;
    b.X = V; b.rows = n; b.K = n; b.si = 1; b.sk = m; b.I = n; b.conj = 1;
    zproduct(ctx, zgemm_params(OP_N, OP_C, n, n, n, T, n, V, m, Z, n), a, b, n, 0, n, true);
    a.X = V; a.rows = m; a.K = n; a.si = 1; a.sk = m; a.I = m; a.conj = 0;
    b.X = Z; b.rows = n; b.K = n; b.si = n; b.sk = 1; b.I = n; b.conj = 0;
    zproduct(ctx, zgemm_params(OP_N, OP_N, m, n, n, V, m, Z, n, Q, m), a, b, m, 0, m, true);
    one_minus_kernel<<<gsz((long long)m * n), 256, 0, ctx.stream>>>(m, n, Q);
    NC_CHECK_LAUNCH();
    ctx.launches++;
}

double qr_plan_bytes(int m, int n) {
    const double k = n, chunks = (m + kDotChain - 1) / kDotChain;
    double q = 0;   // Q's products where they are part of the graph: T V_1^H and split-K partials
    if (residue_scratch_bytes(n, n, n) + residue_scratch_bytes(m, n, n) == 0)
        q = sizeof(cplx) * k * k +
            (double)std::max(zgemm_workspace_bytes(zgemm_params(OP_N, OP_C, n, n, n, nullptr, n, nullptr, m, nullptr, n)),
                             zgemm_workspace_bytes(zgemm_params(OP_N, OP_N, m, n, n, nullptr, m, nullptr, n, nullptr, m)));
    const double panel = 2.0 * NB * NB * ((n + NB - 1) / NB) + 2.0 * NB * NB * (chunks + 1);   // per block; partials and one T
    return sizeof(cplx) * (3.0 * m * k + 2.0 * k * k + (2.0 * NB + 1) * k + panel) + q + 16384.0;
}

double qr_scratch_bytes(int m, int n) {
    const double k = n, chunks = (m + kDotChain - 1) / kDotChain;
    return sizeof(cplx) * (k * k + NB * k * chunks) + std::max(residue_scratch_bytes(n, n, n), residue_scratch_bytes(m, n, n));
}

// ---------------------------------------------------------------------------
// gauge moves (core.f95:2708-2960 semantics, QR gauge)
// ---------------------------------------------------------------------------

// A QR of one shape recorded as a CUDA graph: a gauge move issues a few
// hundred short kernels (the panels are latency bound), so replaying a
// pre-recorded graph removes the per-launch host overhead.  The plan owns its
// input/output buffers and a private workspace arena, so the pointers baked
// into the graph stay valid and are never shared with other work.  Q's products
// are part of the graph unless their integers need scratch of several times the
// matrix: then they follow it, with the context's scratch, which every shape shares.
struct QrPlan {
    const Context* owner = nullptr;   // its graph reports expired waits to this context
    int m = 0, n = 0;
    bool conjR = false;
    Arena arena = Arena::exact();
    // look-ahead: the thread's second stream (side_context, whose arena every
    // plan's graph uses) and the plan's events
    bool lookahead = false;
    std::vector<cudaEvent_t> ev;
    // single-block shapes are run directly: recording a graph saves nothing
    bool capture = true;
    cplx* X = nullptr;   // input (m x n), overwritten
    cplx* Q = nullptr;   // explicit Q (m x n)
    cplx* R = nullptr;   // R (n x n), conjugated if conjR
    cplx* V = nullptr;   // reflectors (m x n) and compact-WY factor (n x n), look-ahead form only
    cplx* T = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    uint64_t kernels = 0;
    ~QrPlan() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        for (cudaEvent_t e : ev) cudaEventDestroy(e);
    }
};

namespace {
// Second stream of this host thread for the look-ahead QR (one per thread,
// shared by the thread's plans, which run one at a time).
Context& side_context() {
    thread_local Context* c = new Context();   // lives until process exit, like Context::get()
    return *c;
}

QrPlan& qr_plan(Context& ctx, int m, int n, bool conjR) {
    thread_local std::vector<std::unique_ptr<QrPlan>> plans;
    for (auto& p : plans)
        if (p->owner == &ctx && p->m == m && p->n == n && p->conjR == conjR) return *p;
    auto p = std::make_unique<QrPlan>();
    p->owner = &ctx;
    p->m = m; p->n = n; p->conjR = conjR;
    p->arena.reserve((size_t)qr_plan_bytes(m, n));
    p->X = p->arena.alloc_n<cplx>((size_t)m * n);
    p->Q = p->arena.alloc_n<cplx>((size_t)m * n);
    p->R = p->arena.alloc_n<cplx>((size_t)n * n);
    if (cluster_qr_available()) {
        p->lookahead = true;
        p->ev.resize(4 + 2 * ((n + NB - 1) / NB));   // the last two fork/join the priority stream
        for (cudaEvent_t& e : p->ev) NC_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    p->capture = n > NB;
    if (p->lookahead && p->capture) {
        p->V = p->arena.alloc_n<cplx>((size_t)m * n);
        p->T = p->arena.alloc_n<cplx>((size_t)n * n);
    }
    plans.push_back(std::move(p));
    return *plans.back();
}

// Highest-priority stream of this host thread for the critical path of the
// recorded look-ahead QR (panels, T, next-block updates).  Graph nodes keep
// the priority of the stream they were captured from (the graph is
// instantiated with cudaGraphInstantiateFlagUseNodePriority), so a pending
// cluster launch is dispatched ahead of the trailing-update GEMMs of the
// second stream as SMs drain.  Null when the stream cannot be created.
cudaStream_t priority_stream() {
    thread_local cudaStream_t s = [] {
        int least = 0, greatest = 0;
        cudaStream_t st = nullptr;
        if (cudaDeviceGetStreamPriorityRange(&least, &greatest) != cudaSuccess ||
            cudaStreamCreateWithPriority(&st, cudaStreamNonBlocking, greatest) != cudaSuccess) {
            cudaGetLastError();
            st = nullptr;
        }
        return st;
    }();
    return s;
}

bool q_after(const QrPlan& P) { return residue_gemm_pays(P.n, P.n, P.n) || residue_gemm_pays(P.m, P.n, P.n); }

// Records `once` as the plan's graph.  The result is there already, so a recording
// that fails costs the graph only, and the next call tries again: the legacy
// default stream cannot be recorded, and another thread's device-wide
// synchronisation ends a recording.
template <typename F>
void record_qr(Context& ctx, QrPlan& P, F& once) {
    const uint64_t l0 = ctx.launches;
    const cudaStream_t home = ctx.stream;
    const cudaStream_t hp = P.lookahead ? priority_stream() : nullptr;
    cudaGraph_t graph = nullptr;
    if (cudaStreamBeginCapture(home, cudaStreamCaptureModeRelaxed) == cudaSuccess) {
        bool whole = false;
        try {
            if (hp) {
                NC_CUDA(cudaEventRecord(P.ev[P.ev.size() - 2], home));
                NC_CUDA(cudaStreamWaitEvent(hp, P.ev[P.ev.size() - 2], 0));
                ctx.stream = hp;
            }
            once();
            if (hp) {
                NC_CUDA(cudaEventRecord(P.ev[P.ev.size() - 1], hp));
                NC_CUDA(cudaStreamWaitEvent(home, P.ev[P.ev.size() - 1], 0));
            }
            whole = true;
        } catch (...) {
        }
        ctx.stream = home;
        if (cudaStreamEndCapture(home, &graph) != cudaSuccess) graph = nullptr;
        if (graph && whole && cudaGraphInstantiateWithFlags(&P.exec, graph, cudaGraphInstantiateFlagUseNodePriority) == cudaSuccess) {
            P.graph = graph;
            P.kernels = ctx.launches - l0;
        } else {
            P.exec = nullptr;
            if (graph) cudaGraphDestroy(graph);
        }
    }
    cudaGetLastError();
    ctx.launches = l0;
}

// Run the QR of plan.X; the first run of a shape executes directly (so the
// private arena grows to its final size) and then records the graph.
void qr_run(Context& ctx, QrPlan& P) {
    if (P.exec) {
        NC_CUDA(cudaGraphLaunch(P.exec, ctx.stream));
        ctx.launches += P.kernels;
        if (P.lookahead && q_after(P)) qr_form_q(ctx, P.m, P.n, P.V, P.T, P.Q);
        return;
    }
    const bool prof = ctx.profile;
    ctx.profile = false;
    ctx.ws_override = &P.arena;
    Context& side = side_context();
    auto once = [&] {
        if (P.lookahead && P.capture) {
            householder_qr_lookahead(ctx, side, P.ev.data(), P.m, P.n, P.X, P.V, P.T, P.R, P.conjR);
            if (!q_after(P)) qr_form_q(ctx, P.m, P.n, P.V, P.T, P.Q);
        } else
            householder_qr(ctx, P.m, P.n, P.X, P.Q, P.R, P.conjR);
    };
    try {
        once();
    } catch (...) {
        ctx.ws_override = nullptr;
        ctx.profile = prof;
        throw;
    }
    if (P.capture) record_qr(ctx, P, once);
    ctx.ws_override = nullptr;
    ctx.profile = prof;
    if (P.lookahead && P.capture && q_after(P)) qr_form_q(ctx, P.m, P.n, P.V, P.T, P.Q);
}
}  // namespace

// The absorption GEMM of the gauge factor, on ctx.stream or, with `as`, on
// the second stream after the QR that produced the factor: there it takes the
// second context's scratch (no QR runs beside it) and reports to ctx.
static void absorb_factor(Context& ctx, const ZGemmParams& p, const ResMatrix& a, const ResMatrix& b, int I,
                          long long sI, long long sn, const AbsorbAsync* as) {
    if (!as) {
        zproduct(ctx, p, a, b, I, sI, sn);
        return;
    }
    NC_CUDA(cudaEventRecord(as->ready, ctx.stream));
    NC_CUDA(cudaStreamWaitEvent(as->stream, as->ready, 0));
    if (residue_gemm_pays(a.rows, b.rows, a.K)) {
        struct OnStream {   // the second context's work on another stream, for the life of this object
            Context& c;
            cudaStream_t s;
            DeviceWatch* w;
            OnStream(Context& side, const Context& ctx, cudaStream_t on) : c(side), s(side.stream), w(side.watch) {
                c.stream = on;
                c.watch = ctx.watch;
            }
            ~OnStream() { c.stream = s; c.watch = w; }
        } on(side_context(), ctx, as->stream);
        const uint64_t l0 = on.c.launches;
        zproduct(on.c, p, a, b, I, sI, sn);
        ctx.launches += on.c.launches - l0;
    } else {
        zgemm(p, as->stream);
        ctx.launches++;
    }
    NC_CUDA(cudaEventRecord(as->done, as->stream));
}

void gauge_right(Context& ctx, int bl, int bm, int br, int dl, int dr, const cplx* A, const cplx* B,
                 cplx* normA, cplx* denormB, const AbsorbAsync* async) {
    const int K = bl * dl;
    NC_ARG(K >= bm, "not enough degrees of freedom to normalize");
    QrPlan& P = qr_plan(ctx, K, bm, false);
    const int p_t[3] = {1, 0, 2};
    permute3(ctx, A, bm, K, 1, p_t, true, P.X);             // X = A^H  (K x bm)
    qr_run(ctx, P);                                          // A^H = Qt Rt
    if (B && denormB) {
        // denormB_s = B_s Rt^H  (neighbour absorbs P = Rt^H on its left index)
        ZGemmParams p = zgemm_params(OP_N, OP_C, br, bm, bm, B, br, P.R, bm, denormB, br);
        p.batch = dr;
        p.sA0 = (long long)br * bm; p.sB0 = 0; p.sC0 = (long long)br * bm;
        ResMatrix a, b;   // rows (r, s) of B against the rows of conj(Rt)
        a.X = B; a.rows = br * dr; a.K = bm; a.si = 1; a.I = br; a.sI = (long long)br * bm; a.sk = br;
        b.X = P.R; b.rows = bm; b.K = bm; b.si = 1; b.I = bm; b.sk = bm; b.conj = 1;
        absorb_factor(ctx, p, a, b, br, (long long)br * bm, br, async);
    }
    permute3(ctx, P.Q, K, bm, 1, p_t, true, normA);         // normA = Qt^H
}

void gauge_left(Context& ctx, int bl, int bm, int br, int dl, int dr, const cplx* A, const cplx* B,
                cplx* denormA, cplx* normB, const AbsorbAsync* async) {
    const int K = br * dr;
    NC_ARG(K >= bm, "not enough degrees of freedom to normalize");
    QrPlan& P = qr_plan(ctx, K, bm, true);
    const cplx* Rc = P.R;
    const int p_rs[3] = {0, 2, 1};
    permute3(ctx, B, br, bm, dr, p_rs, true, P.X);           // X((r,s),m) = conj(B(r,m,s))
    qr_run(ctx, P);                                          // Rc = conj(Rt)
    if (A && denormA) {
        // denormA = conj(Rt) * A  (as bm x bl*dl)
        ResMatrix a, b;
        a.X = Rc; a.rows = bm; a.K = bm; a.si = 1; a.I = bm; a.sk = bm;
        b.X = A; b.rows = bl * dl; b.K = bm; b.si = bm; b.I = b.rows; b.sk = 1;
        absorb_factor(ctx, zgemm_params(OP_N, OP_N, bm, bl * dl, bm, Rc, bm, A, bm, denormA, bm), a, b, bm, 0, bm, async);
    }
    permute3(ctx, P.Q, br, dr, bm, p_rs, true, normB);       // normB(r,m,s) = conj(Qt((r,s),m))
}

void rand_norm_site(Context& ctx, int br, int bl, int d, uint64_t seed, cplx* out) {
    // core.f95:2634-2659: columns l of the (br*d x bl) workspace orthonormal
    NC_ARG(br * d >= bl, "not enough degrees of freedom to normalize");
    ArenaFrame f(ctx.arena);
    const int K = br * d;
    cplx* X = ctx.arena.alloc_n<cplx>((size_t)K * bl);
    cplx* Qt = ctx.arena.alloc_n<cplx>((size_t)K * bl);
    zrandom(ctx, (long long)K * bl, seed, X);
    householder_qr(ctx, K, bl, X, Qt, nullptr, false);
    const int p_rs[3] = {0, 2, 1};
    permute3(ctx, Qt, br, d, bl, p_rs, false, out);  // state(r,l,s) = ws(r,s,l)
}

void rand_unnorm_site(Context& ctx, int br, int bl, int d, uint64_t seed, cplx* out) {
    // core.f95:2661-2671
    const long long n = (long long)br * bl * d;
    zrandom(ctx, n, seed, out);
    ArenaFrame f(ctx.arena);
    cplx* nr = ctx.arena.alloc_n<cplx>(1);
    znrm2sq(ctx, n, out, nr);
    znormalize_dev(ctx, n, nr, out);
}

void increase_bandwidth(Context& ctx, int bl, int bm, int br, int dl, int dr, int new_bm, uint64_t seed,
                        const cplx* A, const cplx* B, cplx* outA, cplx* outB) {
    // core.f95:3090-3144
    ArenaFrame f(ctx.arena);
    cplx* M = ctx.arena.alloc_n<cplx>((size_t)new_bm * bm);
    cplx* X = ctx.arena.alloc_n<cplx>((size_t)new_bm * bm);
    zrandom(ctx, (long long)new_bm * bm, seed, X);
    householder_qr(ctx, new_bm, bm, X, M, nullptr, false);   // isometry new_bm x bm
    cplx* e1 = ctx.arena.alloc_n<cplx>((size_t)new_bm * bl * dl);
    cplx* e2 = ctx.arena.alloc_n<cplx>((size_t)br * new_bm * dr);
    zgemm(zgemm_params(OP_N, OP_N, new_bm, bl * dl, bm, M, new_bm, A, bm, e1, new_bm), ctx);
    ZGemmParams p = zgemm_params(OP_N, OP_C, br, new_bm, bm, B, br, M, new_bm, e2, br);
    p.batch = dr;
    p.sA0 = (long long)br * bm; p.sB0 = 0; p.sC0 = (long long)br * new_bm;
    zgemm(p, ctx);
    gauge_left(ctx, bl, new_bm, br, dl, dr, e1, e2, outA, outB);
}

}  // namespace nc

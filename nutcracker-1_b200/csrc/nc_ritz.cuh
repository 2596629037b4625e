// Projected (Rayleigh-Ritz) problem of the restarted Lanczos solvers, shared
// by the single-chain solver (lanczos.cu) and the batched one (batched.cu).
//
// T = V^H H V grows by one column per Lanczos step (real symmetric: a
// tridiagonal block plus, after a thick restart, an arrow of couplings to the
// kept Ritz vectors; both come out of the reorthogonalisation coefficients,
// T(i, m-1) = Re(h1_i + h2_i)).  Its eigen-decomposition T = Z Theta Z^T is
// kept between steps (the rotated matrix A ~ Theta and the accumulated
// rotations Z, row-major [row][col], MAXT x MAXT each): a new column t is
// taken into the current eigenbasis (z = Z^T t), which leaves a diagonal
// matrix bordered by one row and column, and one block finishes it with
// cyclic Jacobi (round-robin pairing, which keeps clustered Ritz values such
// as near-degenerate doublets orthogonal).  Started from an almost diagonal
// matrix, Jacobi needs a few sweeps instead of the 6-10 of a cold start; a
// rotation is skipped when its off-diagonal element is below the rounding
// level of its diagonal pair, and the sweeps stop when a sweep would skip
// every rotation.
//
// What bounds it is latency: a sweep is m - 1 rounds, each round's rotation
// angles need the blocks that the round before rotated, and a solve waits for
// it at every Lanczos step.  So the block splits a round over its threads, with
// one barrier a round:
//   warp 0 has the angles of round s and rotates just the three elements a pair
//   of round s + 1 needs, then computes that pair's angles;
//   the other warps meanwhile apply round s: every 2 x 2 block (pair r, pair q)
//   of A, from one copy of A into the other, and every (row, pair) of Z belong
//   to one thread, the same in every round.
// An element that is computed in both places goes through the same operations,
// written with their roundings, and every element of A and Z through those of a
// one-warp update in the same order, so the Ritz pairs are the same bits for
// any number of threads.  Whether a sweep is needed at all is asked of all pairs
// at once instead of by a last sweep that rotates nothing.
// Measured on a B200: one warp 148 us an update (mean over the solve of a
// 48 x 48 x 2 site, 24-vector basis); 65 us, or 2280 clocks a round at m = 24
// and 1950 at m = 20, with A and Z rotated between one round's angles and the
// next's; 1550 and 1510 with Z beside the next angles; now 1430 and 1400.  The
// angles' three divisions and two square roots in a row are 570 of them.
// Starting them from FP32 values with FP64 Newton steps gains another 3% of a
// solve and changes the rounding, so it is not done.
#pragma once

#include "nc_common.cuh"

namespace nc {

enum RitzWhich { RITZ_SR = 0, RITZ_LR = 1, RITZ_LM = 2 };

struct RitzResult {
    double theta, res, beta, tnorm;
    int sweeps;
};

constexpr int RITZ_THREADS = 256;

// Shared-memory work area of one block's update.
template <int MAXT>
struct RitzSmem {
    double A[2][MAXT][MAXT + 1];   // before and after a round
    double Z[MAXT][MAXT + 1];
    double tcol[MAXT];
    double cs[2][MAXT / 2], sn[2][MAXT / 2];   // angles of a round and of the one before
    int perm[MAXT];
};

// Whether the pair (app, aqq) still needs its rotation: apq above the
// rounding level of the pair, |apq| > 2^-53 sqrt(|app| |aqq|).
__device__ __forceinline__ bool ritz_rotates(double apq, double app, double aqq) {
    const double x = fabs(apq);
    if (!(x > 1e-300)) return false;
    if (x > 1e-140 && x < 1e140) {
        const double g = fabs(app) * fabs(aqq);
        if (g < 1e300) return x * x > 1.232595164407831e-32 * g;
    }
    return x > 1.1102230246251565e-16 * sqrt(fabs(app)) * sqrt(fabs(aqq));
}

// The Jacobi rotation that annihilates apq: t = sign(tau) / (|tau| +
// sqrt(1 + tau^2)), tau = (aqq - app) / (2 apq), c = 1 / sqrt(1 + t^2), s = t c.
__device__ __forceinline__ void ritz_rotation(double apq, double app, double aqq, double& c, double& sv) {
    const double tau = (aqq - app) / (2.0 * apq);
    const double t = (tau >= 0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
    c = 1.0 / sqrt(1.0 + t * t);
    sv = t * c;
}

// c x - s y and s x + c y with the roundings spelled out: an element of A is
// computed twice, by the block's owner and for the next angles.  A pair that is
// not rotated (s = 0) keeps its elements, non-finite neighbours or not.
__device__ __forceinline__ double ritz_first(double c, double s, double x, double y) {
    return s == 0.0 ? x : __fma_rn(c, x, -__dmul_rn(s, y));
}
__device__ __forceinline__ double ritz_second(double c, double s, double x, double y) {
    return s == 0.0 ? y : __fma_rn(s, x, __dmul_rn(c, y));
}

// After a thick restart: A = diag(theta_0 .. theta_{k-1}), Z = I.  Any
// number of threads of one block.
template <int MAXT>
__device__ __forceinline__ void ritz_restart_state(int k, const double* theta, double* state) {
    double* A = state;
    double* Z = state + MAXT * MAXT;
    for (int e = threadIdx.x; e < MAXT * MAXT; e += blockDim.x) {
        const int r = e / MAXT, c = e % MAXT;
        A[e] = (r == c && r < k) ? theta[r] : 0.0;
        Z[e] = (r == c) ? 1.0 : 0.0;
    }
}

// One block of RITZ_THREADS threads (MAXT <= 32): adds column m-1 of T
// (tcol(i) = Re(h1_i + h2_i), i < m) to the kept decomposition of the leading
// (m-1) x (m-1) block in `state` and diagonalises.  The Ritz values, ordered
// by `which` (SR ascending, LR descending, LM by decreasing magnitude), go to
// theta[], the matching eigenvectors of T to S (column r at S[ldS * r], m
// entries; complex with zero imaginary part when S_complex, else real).  The
// wanted pair's value and Ritz estimate beta |z_{m-1,0}| (beta =
// sqrt(nrm2)) are returned to every thread.
template <int MAXT, bool S_complex>
__device__ RitzResult ritz_update_block(RitzSmem<MAXT>& w, int m, double* __restrict__ state,
                                        const cplx* __restrict__ h1, const cplx* __restrict__ h2, double nrm2,
                                        int which, void* __restrict__ S_out, int ldS, double* __restrict__ theta) {
    static_assert(MAXT <= 32, "one warp computes the angles and the border");
    const int tid = threadIdx.x;
    const int mp = m + (m & 1), np = mp / 2;
    int cur = 0;   // the valid half of w.A
    // load the kept (m-1) x (m-1) decomposition, pad to mp
    for (int e = tid; e < mp * MAXT; e += RITZ_THREADS) {
        const int r = e / MAXT, q = e % MAXT;
        const bool in = q < m - 1 && r < m - 1;
        w.A[0][r][q] = in ? state[e] : 0.0;
        w.Z[r][q] = in ? state[MAXT * MAXT + e] : (r == q ? 1.0 : 0.0);
    }
    if (tid < m) w.tcol[tid] = h1[tid].x + h2[tid].x;
    __syncthreads();
    // border: z = Z^T t over the old rows, diagonal t_{m-1}
    if (tid < m - 1) {
        double z = 0.0;
        for (int i = 0; i < m - 1; ++i) z += w.Z[i][tid] * w.tcol[i];
        w.A[0][tid][m - 1] = z;
        w.A[0][m - 1][tid] = z;
    }
    if (tid == 0) w.A[0][m - 1][m - 1] = w.tcol[m - 1];
    __syncthreads();
    // Thread-constant work: elements of the check; blocks of A and (row, pair)s of Z (warps 1 ..).
    constexpr int WT = RITZ_THREADS - 32;
    constexpr int NCHK = (MAXT * MAXT / 2 + RITZ_THREADS - 1) / RITZ_THREADS;
    constexpr int NBLK = (MAXT * MAXT / 4 + WT - 1) / WT, NROT = (MAXT * MAXT / 2 + WT - 1) / WT;
    int ca[NCHK], cb[NCHK], blk_r[NBLK], blk_q[NBLK], zi[NROT], zq[NROT];
#pragma unroll
    for (int u = 0; u < NCHK; ++u) {
        const int e = tid + u * RITZ_THREADS, s = e / np, r = e - s * np;
        ca[u] = r == 0 ? mp - 1 : (s + r) % (mp - 1);
        cb[u] = s >= mp - 1 ? -1 : r == 0 ? s : (s - r + mp - 1) % (mp - 1);
    }
#pragma unroll
    for (int u = 0; u < NBLK; ++u) {
        const int f = tid - 32 + u * WT;
        blk_r[u] = f >= 0 ? f / np : np;
        blk_q[u] = f - blk_r[u] * np;
    }
#pragma unroll
    for (int u = 0; u < NROT; ++u) {
        const int f = tid - 32 + u * WT;
        zi[u] = f >= 0 ? f / np : m;
        zq[u] = f - zi[u] * np;
    }
    // round s's pairs: r = 0 (mp-1, s), r > 0 (s + r, s - r) mod mp-1
    auto first = [&](int s, int r) { const int a = s + r; return r == 0 ? mp - 1 : (a >= mp - 1 ? a - (mp - 1) : a); };
    auto second = [&](int s, int r) { const int b = s - r; return r == 0 ? s : (b < 0 ? b + (mp - 1) : b); };
    // Where pair `tid` of a round comes from: its first index is member ma of
    // pair pa of the round before, its second index member mb of pair pb.
    const int pa = tid == 0 ? 0 : min(tid + 1, np - 1), pb = tid == 0 ? min(1, np - 1) : tid - 1;
    const bool ma = tid > 0 && tid == np - 1, mb = tid > 0;
    auto angles = [&](int slot, double apq, double app, double aqq) {
        double c = 1.0, sv = 0.0;
        if (ritz_rotates(apq, app, aqq)) ritz_rotation(apq, app, aqq, c, sv);
        w.cs[slot][tid] = c;
        w.sn[slot][tid] = sv;
    };
    int sweep = 0;
    for (; sweep < 30; ++sweep) {
        bool any = false;   // a sweep is needed while any pair would rotate; asked of the same element as in its round
        const double(&A0)[MAXT][MAXT + 1] = w.A[cur];
#pragma unroll
        for (int u = 0; u < NCHK; ++u)
            if (cb[u] >= 0) any |= ritz_rotates(A0[ca[u]][cb[u]], A0[ca[u]][ca[u]], A0[cb[u]][cb[u]]);
        if (!__syncthreads_or(any)) break;
        if (tid < np) {
            const int a = first(0, tid), b = second(0, tid);
            angles(0, A0[a][b], A0[a][a], A0[b][b]);
        }
        __syncthreads();
        for (int s = 0; s < mp - 1; ++s) {
            const double(&A)[MAXT][MAXT + 1] = w.A[cur];
            const double *cs = w.cs[s & 1], *sn = w.sn[s & 1];
            if (tid < np) {
                if (s < mp - 2) {   // the next round's angles, from this round's rotation of the elements they need
                    const int a0 = first(s, pa), a1 = second(s, pa), b0 = first(s, pb), b1 = second(s, pb);
                    const double ac = cs[pa], as = sn[pa], bc = cs[pb], bs = sn[pb];
                    // ritz_first or ritz_second by the member, as one expression
                    const double a_x = ma ? as : ac, a_y = ma ? ac : -as, b_x = mb ? bs : bc, b_y = mb ? bc : -bs;
                    const bool a_rot = as != 0.0, b_rot = bs != 0.0;
                    auto mix_a = [&](double x, double y) {
                        const double v = __fma_rn(a_x, x, __dmul_rn(a_y, y));
                        return a_rot ? v : ma ? y : x;
                    };
                    auto mix_b = [&](double x, double y) {
                        const double v = __fma_rn(b_x, x, __dmul_rn(b_y, y));
                        return b_rot ? v : mb ? y : x;
                    };
                    const double p00 = A[a0][b0], p01 = A[a0][b1], p10 = A[a1][b0], p11 = A[a1][b1];
                    const double u00 = A[a0][a0], u01 = A[a0][a1], u10 = A[a1][a0], u11 = A[a1][a1];
                    const double v00 = A[b0][b0], v01 = A[b0][b1], v10 = A[b1][b0], v11 = A[b1][b1];
                    const double apq = mix_b(mix_a(p00, p10), mix_a(p01, p11));
                    const double app = mix_a(mix_a(u00, u10), mix_a(u01, u11));
                    const double aqq = mix_b(mix_b(v00, v10), mix_b(v01, v11));
                    angles((s + 1) & 1, apq, app, aqq);
                }
            } else if (tid >= 32) {
                double(&B)[MAXT][MAXT + 1] = w.A[cur ^ 1];
#pragma unroll
                for (int u = 0; u < NBLK; ++u) {   // block (rows of pair r, columns of pair q)
                    const int r = blk_r[u], q = blk_q[u];
                    if (r >= np) continue;
                    const double cr = cs[r], sr = sn[r], cq = cs[q], sq = sn[q];
                    const int ar = first(s, r), br = second(s, r), aq = first(s, q), bq = second(s, q);
                    const double x00 = A[ar][aq], x01 = A[ar][bq], x10 = A[br][aq], x11 = A[br][bq];
                    const double y00 = ritz_first(cr, sr, x00, x10), y01 = ritz_first(cr, sr, x01, x11);
                    const double y10 = ritz_second(cr, sr, x00, x10), y11 = ritz_second(cr, sr, x01, x11);
                    B[ar][aq] = ritz_first(cq, sq, y00, y01);
                    B[ar][bq] = ritz_second(cq, sq, y00, y01);
                    B[br][aq] = ritz_first(cq, sq, y10, y11);
                    B[br][bq] = ritz_second(cq, sq, y10, y11);
                }
#pragma unroll
                for (int u = 0; u < NROT; ++u) {   // columns of pair q in row i of Z
                    if (zi[u] >= m) continue;
                    const int i = zi[u], q = zq[u], a = first(s, q), b = second(s, q);
                    const double c = cs[q], sv = sn[q], va = w.Z[i][a], vb = w.Z[i][b];
                    if (sv == 0.0) continue;
                    w.Z[i][a] = ritz_first(c, sv, va, vb);
                    w.Z[i][b] = ritz_second(c, sv, va, vb);
                }
            }
            __syncthreads();
            cur ^= 1;
        }
    }
    __syncthreads();
    const double(&A)[MAXT][MAXT + 1] = w.A[cur];
    // order the m genuine Ritz values by rank (a padding direction, if any, is index m)
    if (tid < m) w.perm[tid] = tid;
    __syncthreads();
    int rank = 0;
    if (tid < m) {
        const double x = A[tid][tid];
        for (int q = 0; q < m; ++q) {
            const double y = A[q][q];
            const bool better = (which == RITZ_SR) ? (y < x) : (which == RITZ_LR) ? (y > x) : (fabs(y) > fabs(x));
            const bool worse = (which == RITZ_SR) ? (x < y) : (which == RITZ_LR) ? (x > y) : (fabs(x) > fabs(y));
            rank += (better || (!worse && q < tid)) ? 1 : 0;
        }
    }
    __syncthreads();
    if (tid < m) w.perm[rank] = tid;
    __syncthreads();
    // keep the decomposition of the m x m block for the next step, and the ordered pairs
    for (int e = tid; e < m * MAXT; e += RITZ_THREADS) {
        const int r = e / MAXT, q = e % MAXT;
        if (q >= m) continue;
        state[e] = A[r][q];
        state[MAXT * MAXT + e] = w.Z[r][q];
        const double z = w.Z[q][w.perm[r]];
        if (S_complex) reinterpret_cast<cplx*>(S_out)[q + (size_t)ldS * r] = cmake(z, 0.0);
        else reinterpret_cast<double*>(S_out)[q + (size_t)ldS * r] = z;
    }
    if (tid < m) theta[tid] = A[w.perm[tid]][w.perm[tid]];
    RitzResult out{};
    double tn = 0;
    for (int i = 0; i < m; ++i) tn = fmax(tn, fabs(A[i][i]));
    const double beta = sqrt(nrm2);
    out.theta = A[w.perm[0]][w.perm[0]];
    out.res = beta * fabs(w.Z[m - 1][w.perm[0]]);
    out.beta = beta;
    out.tnorm = tn;
    out.sweeps = sweep;
    return out;
}

}  // namespace nc

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
// What bounds it is latency: a sweep is m - 1 rounds, each the chain
// (rotation angles) -> (rotated blocks of A), and a solve waits for it at
// every Lanczos step.  So the block splits each round over its threads: one
// warp computes the angles of the round's disjoint pairs while the others
// apply the round before to Z, which no angle depends on; then every 2 x 2
// block (pair r, pair q) of A belongs to one thread, in place.  Which block,
// rows and pairs a thread has is the same in every round and computed once.
// Whether a sweep is needed at all is asked of all pairs at once instead of by
// a last sweep that rotates nothing.  Every element goes through the same
// operations in the same order as in a one-warp update, so the Ritz pairs are
// the same bits for any number of threads.  Measured on a B200: one warp
// 148 us an update (mean over the solve of a 48 x 48 x 2 site, 24-vector
// basis), 65 us with A and Z rotated together between the angles, that is
// 2280 clocks a round at m = 24 and 1950 at m = 20, now 1550 and 1510; most of
// that is the angles' three divisions and two square roots in a row.
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
    double A[MAXT][MAXT + 1], Z[MAXT][MAXT + 1];
    double tcol[MAXT];
    double cs[2][MAXT / 2], sn[2][MAXT / 2];   // angles of a round and of the one before
    int perm[MAXT];
    int rotated[2];
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
    // load the kept (m-1) x (m-1) decomposition, pad to mp
    for (int e = tid; e < mp * MAXT; e += RITZ_THREADS) {
        const int r = e / MAXT, q = e % MAXT;
        const bool in = q < m - 1 && r < m - 1;
        w.A[r][q] = in ? state[e] : 0.0;
        w.Z[r][q] = in ? state[MAXT * MAXT + e] : (r == q ? 1.0 : 0.0);
    }
    if (tid < m) w.tcol[tid] = h1[tid].x + h2[tid].x;
    __syncthreads();
    // border: z = Z^T t over the old rows, diagonal t_{m-1}
    if (tid < m - 1) {
        double z = 0.0;
        for (int i = 0; i < m - 1; ++i) z += w.Z[i][tid] * w.tcol[i];
        w.A[tid][m - 1] = z;
        w.A[m - 1][tid] = z;
    }
    if (tid == 0) w.A[m - 1][m - 1] = w.tcol[m - 1];
    __syncthreads();
    // Thread-constant work: elements of the check, one block of A, (row, pair) of Z.
    static_assert(MAXT * MAXT / 4 <= RITZ_THREADS, "one block of A per thread");
    constexpr int NCHK = (MAXT * MAXT / 2 + RITZ_THREADS - 1) / RITZ_THREADS;
    constexpr int ZT = RITZ_THREADS - 32, NROT = (MAXT * MAXT / 2 + ZT - 1) / ZT;
    int ca[NCHK], cb[NCHK], zi[NROT], zq[NROT];
#pragma unroll
    for (int u = 0; u < NCHK; ++u) {
        const int e = tid + u * RITZ_THREADS, s = e / np, r = e - s * np;
        ca[u] = r == 0 ? mp - 1 : (s + r) % (mp - 1);
        cb[u] = s >= mp - 1 ? -1 : r == 0 ? s : (s - r + mp - 1) % (mp - 1);
    }
#pragma unroll
    for (int u = 0; u < NROT; ++u) {
        const int f = tid - 32 + u * ZT;
        zi[u] = f >= 0 ? f / np : m;
        zq[u] = f - zi[u] * np;
    }
    const int rA = tid / np, qA = tid - rA * np;
    // round s's pairs: r = 0 (mp-1, s), r > 0 (s + r, s - r) mod mp-1
    auto first = [&](int s, int r) { const int a = s + r; return r == 0 ? mp - 1 : (a >= mp - 1 ? a - (mp - 1) : a); };
    auto second = [&](int s, int r) { const int b = s - r; return r == 0 ? s : (b < 0 ? b + (mp - 1) : b); };
    // columns of pair q in row i of Z, round s
    auto rotate_z = [&](int s) {
        if (!w.rotated[s & 1]) return;
#pragma unroll
        for (int u = 0; u < NROT; ++u) {
            if (zi[u] >= m) continue;
            const int i = zi[u], a = first(s, zq[u]), b = second(s, zq[u]);
            const double cq = w.cs[s & 1][zq[u]], sq = w.sn[s & 1][zq[u]], va = w.Z[i][a], vb = w.Z[i][b];
            if (sq == 0.0) continue;
            w.Z[i][a] = cq * va - sq * vb;
            w.Z[i][b] = sq * va + cq * vb;
        }
    };
    int sweep = 0;
    for (; sweep < 30; ++sweep) {
        bool any = false;   // a sweep is needed while any pair would rotate; asked of the same element as in its round
#pragma unroll
        for (int u = 0; u < NCHK; ++u)
            if (cb[u] >= 0) any |= ritz_rotates(w.A[ca[u]][cb[u]], w.A[ca[u]][ca[u]], w.A[cb[u]][cb[u]]);
        if (!__syncthreads_or(any)) break;
        for (int s = 0; s < mp - 1; ++s) {
            if (tid < 32) {
                double c = 1.0, sv = 0.0;
                bool rot = false;
                if (tid < np) {
                    const int a = first(s, tid), b = second(s, tid);
                    const double apq = w.A[a][b], app = w.A[a][a], aqq = w.A[b][b];
                    rot = ritz_rotates(apq, app, aqq);
                    if (rot) ritz_rotation(apq, app, aqq, c, sv);
                    w.cs[s & 1][tid] = c;
                    w.sn[s & 1][tid] = sv;
                }
                rot = __any_sync(0xffffffffu, rot);
                if (tid == 0) w.rotated[s & 1] = rot;
            } else if (s > 0) {
                rotate_z(s - 1);
            }
            __syncthreads();
            if (!w.rotated[s & 1]) continue;
            if (rA < np) {   // block (rows of pair rA, columns of pair qA)
                const double cr = w.cs[s & 1][rA], sr = w.sn[s & 1][rA], cq = w.cs[s & 1][qA], sq = w.sn[s & 1][qA];
                const int ar = first(s, rA), br = second(s, rA), aq = first(s, qA), bq = second(s, qA);
                double x00 = w.A[ar][aq], x01 = w.A[ar][bq], x10 = w.A[br][aq], x11 = w.A[br][bq];
                if (sr != 0.0) {   // rows
                    const double y0 = x00, y1 = x01;
                    x00 = cr * y0 - sr * x10;
                    x01 = cr * y1 - sr * x11;
                    x10 = sr * y0 + cr * x10;
                    x11 = sr * y1 + cr * x11;
                }
                if (sq != 0.0) {   // columns
                    const double y0 = x00, y1 = x10;
                    x00 = cq * y0 - sq * x01;
                    x10 = cq * y1 - sq * x11;
                    x01 = sq * y0 + cq * x01;
                    x11 = sq * y1 + cq * x11;
                }
                w.A[ar][aq] = x00; w.A[ar][bq] = x01; w.A[br][aq] = x10; w.A[br][bq] = x11;
            }
            __syncthreads();
        }
        if (tid >= 32) rotate_z(mp - 2);
    }
    __syncthreads();
    // order the m genuine Ritz values by rank (a padding direction, if any, is index m)
    if (tid < m) w.perm[tid] = tid;
    __syncthreads();
    int rank = 0;
    if (tid < m) {
        const double x = w.A[tid][tid];
        for (int q = 0; q < m; ++q) {
            const double y = w.A[q][q];
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
        state[e] = w.A[r][q];
        state[MAXT * MAXT + e] = w.Z[r][q];
        const double z = w.Z[q][w.perm[r]];
        if (S_complex) reinterpret_cast<cplx*>(S_out)[q + (size_t)ldS * r] = cmake(z, 0.0);
        else reinterpret_cast<double*>(S_out)[q + (size_t)ldS * r] = z;
    }
    if (tid < m) theta[tid] = w.A[w.perm[tid]][w.perm[tid]];
    RitzResult out{};
    double tn = 0;
    for (int i = 0; i < m; ++i) tn = fmax(tn, fabs(w.A[i][i]));
    const double beta = sqrt(nrm2);
    out.theta = w.A[w.perm[0]][w.perm[0]];
    out.res = beta * fabs(w.Z[m - 1][w.perm[0]]);
    out.beta = beta;
    out.tnorm = tn;
    out.sweeps = sweep;
    return out;
}

}  // namespace nc

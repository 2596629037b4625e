// Complex128 GEMM through residues on the int8 tensor cores (sm_100a).
//
// tcgen05 has no FP64 kind, and the FP64 tensor pipe (mma.sync DMMA,
// zgemm.cu) gives 30 TFLOP/s; the int8 kind multiplies about a hundred times
// faster.  So a large product C = A B runs in exact integer arithmetic modulo
// L = 20 small coprime moduli (the "Ozaki scheme II" of Ozaki, Uchino and
// Imamura 2025):
//   1. every row of A and column of B is scaled by a power of two so that its
//      2-norm lies in (2^76, 2^77], and rounded to integers;
//   2. the integers' residues modulo each p_l fit in a byte (planes Re, Im and
//      Re + Im, so that one complex product is three real ones);
//   3. per modulus, three 8-bit GEMMs with int32 accumulation in tensor memory
//      give P1 = Re Re, P2 = Im Im, P3 = (Re + Im)(Re + Im); the epilogue
//      reduces Re C = P1 - P2 and Im C = P3 - P1 - P2 modulo p_l to a byte;
//   4. the Chinese remainder theorem rebuilds each integer of C from its L
//      residues, and the scales are undone.
// By Cauchy-Schwarz |C_mn| <= 2^154 before the scales are undone, and the
// product of the moduli is above 2^155.4, so the residues determine C.
//
// What is rounded.  Step 1 leaves a component as it is when its lowest bit lies
// within 2^-77 of its row's norm: every component above 2^-24 of the norm, and
// smaller ones with fewer bits.  A component below that keeps an error of at
// most 2^-77 of the norm.  The conversion counts such components, and an
// operand with more than one of 2^15 of them (or with any that is not finite)
// is not multiplied here: the GEMM and the CRT kernel return, and the FP64
// product behind them, which returns at once otherwise, runs.  So an operand
// whose rows span too many magnitudes (a contracted bond with weights far
// apart) goes through the same arithmetic as a small product, and infinities
// and NaN reach the outputs that they reach there.  (With 15 moduli and norms
// up to 2^58, half of all components of a random operand were rounded, and
// behind an identity environment a bond with weights 1 to 1e-8 lost its last
// column to 8e-10 of itself.)  Steps 2 and 3 are exact; step 4 rounds once to
// FP64, to at worst 2^-114 |a_m| |b_n|.
//
// Kernels: norms (HBM read), residues (HBM: 16 bytes read, 60 written per
// complex element), the GEMM (tensor-bound), CRT (HBM: 40 bytes read, 16
// written per element).  The GEMM is one persistent CTA per SM over
// (modulus, column tile, row tile) items: a 128 x 256 tile of one plane's
// product at a time (tcgen05.mma.kind::i8, 128 x 256 x 32 per instruction),
// 128-byte K stages through a 4-deep TMA ring, two 256-column accumulators
// in tensor memory that alternate between planes so that the epilogue of one
// overlaps the MMAs of the next.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>

#include "nc_common.cuh"
#include "nc_kernels.h"
#include "nc_tcgen05.cuh"

namespace nc {

namespace {

// ---- moduli and the constants of the Chinese remainder theorem --------------
constexpr int NL = 20;
constexpr int kMod[NL] = {256, 253, 251, 247, 245, 243, 241, 239, 233, 229, 227, 223, 211, 199, 197, 193, 191, 181, 179, 173};
constexpr int kNormBits = 77;         // scaled rows: 2-norm in (2^76, 2^77]
constexpr int kHigh = 115, kMid = 75; // CRT weights split at 2^115 and 2^75

// A product of up to NL moduli.
struct Big {
    unsigned w[6] = {1, 0, 0, 0, 0, 0};
    constexpr void times(unsigned x) {
        unsigned long long c = 0;
        for (int i = 0; i < 6; ++i) {
            c += (unsigned long long)w[i] * x;
            w[i] = (unsigned)c;
            c >>= 32;
        }
    }
    // bits [from, from + count), count <= 53
    constexpr unsigned long long bits(int from, int count) const {
        unsigned long long v = 0;
        for (int i = 0; i < count; ++i) v |= (unsigned long long)((w[(from + i) / 32] >> ((from + i) % 32)) & 1u) << i;
        return v;
    }
};
// (P / p_l) * ((P / p_l)^-1 mod p_l): 1 modulo p_l, 0 modulo the others; P for l = NL
constexpr Big crt_weight(int l) {
    Big b;
    int r = 1;
    for (int i = 0; i < NL; ++i)
        if (i != l) {
            b.times((unsigned)kMod[i]);
            if (l < NL) r = r * kMod[i] % kMod[l];
        }
    if (l < NL) {
        int inv = 1;
        while ((inv * r) % kMod[l] != 1) ++inv;
        b.times((unsigned)inv);
    }
    return b;
}
constexpr double high_part(const Big& b) { return (double)b.bits(kHigh, 192 - kHigh > 53 ? 53 : 192 - kHigh); }
constexpr double mid_part(const Big& b) { return (double)b.bits(kMid, kHigh - kMid); }
constexpr double low_part(const Big& b) { return (double)b.bits(37, kMid - 37) * 137438953472.0 + (double)b.bits(0, 37); }
constexpr int pow2_mod(int e, int p) {
    int r = 1;
    for (int i = 0; i < e; ++i) r = (2 * r) % p;
    return r;
}
constexpr Big kP = crt_weight(NL);
static_assert(kP.bits(2 * kNormBits + 1, 10) == 1, "2 * 2^(2 kNormBits) < P < 2^156");

constexpr float kMagicF = 12582912.0f;      // 1.5 * 2^23: a float added to it is rounded to an integer
constexpr unsigned kMagicI = 0x4B400000u;   // its bits: kMagicI + i is the float kMagicF + i, |i| < 2^22
constexpr int kBias = kNormBits;            // integers are stored plus 2^kBias, so 0 <= v <= 2^78
constexpr int kTop = 48;                    // in three words: v = w2 2^48 + w1 2^32 + w0, w1 < 2^16
struct Tables {
    unsigned p[NL];               // modulus
    float invf[NL], half[NL];     // 1 / p, kMagicF + floor(p / 2)
    unsigned m0[NL], m1[NL], m2[NL];   // 2^(8 i) modulo p for the bytes of the three words, packed
    unsigned off[NL];             // kMagicI + (minus 2^kBias modulo p)
    int inv38[NL];                // 2^38 / p, rounded
    double wh[NL], wm[NL], wl[NL];   // CRT weights: wh 2^115 + wm 2^75 + wl
};
constexpr Tables make_tables() {
    Tables t{};
    for (int l = 0; l < NL; ++l) {
        const int p = kMod[l];
        t.p[l] = (unsigned)p;
        t.invf[l] = 1.0f / (float)p;
        t.half[l] = kMagicF + (float)(p / 2);
        for (int i = 0; i < 4; ++i) {
            t.m0[l] |= (unsigned)(pow2_mod(8 * i, p) & 255) << (8 * i);
            if (i < 2) t.m1[l] |= (unsigned)(pow2_mod(32 + 8 * i, p) & 255) << (8 * i);
            t.m2[l] |= (unsigned)(pow2_mod(kTop + 8 * i, p) & 255) << (8 * i);
        }
        t.off[l] = kMagicI + (unsigned)((p - pow2_mod(kBias, p)) % p);
        t.inv38[l] = (int)(((1ull << 38) + p / 2) / p);
        const Big w = crt_weight(l);
        t.wh[l] = high_part(w);
        t.wm[l] = mid_part(w);
        t.wl[l] = low_part(w);
    }
    return t;
}
constexpr Tables kC = make_tables();
__constant__ Tables kT = make_tables();   // for a modulus known at run time only
constexpr double kPh = high_part(kP), kPm = mid_part(kP), kPl = low_part(kP);
constexpr unsigned long long kNormwise = 1ull << 39;   // limit on rounded components that only a non-finite row exceeds
constexpr int kBadExp = 1 << 30;         // exponent of a row with a non-finite element
constexpr int kMaxK = 16000;             // |Re|, |Im| sums of K residue products fit in int32

// four values' low bytes
__device__ __forceinline__ uint32_t pack4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}

// ---- operands ------------------------------------------------------------------
// Row i, K index k of a complex operand: X[(i % I) * si + (i / I) * sI + k * sk].
struct ResSource {
    const cplx* X;
    long long si, sI, sk;
    int I, rows, K;
    int conj;
};

constexpr int NT = 256;

__device__ __forceinline__ const cplx* row_ptr(const ResSource& s, int i) {
    return s.X + (long long)(i % s.I) * s.si + (long long)(i / s.I) * s.sI;
}

// One launch handles both operands of a product (the first nb[0] blocks along
// x are operand 0's), so that a small product does not wait for two launches.
struct ResPair {
    ResSource s[2];
    double2* part[2];     // [K chunk][row]
    int* exps[2];
    uint8_t* planes[2];
    int nb[2], nchunk[2], chunk[2];
    int Kp, lper;         // padded K; moduli per block
    unsigned long long* rounded;   // per operand: components that step 1 rounds
    unsigned long long limit[2];   // more of them: the product is not made here
};

// A component as the three words of its integer, offset by 2^kBias.
struct Fixed {
    uint32_t w0, w1, w2;
};
__device__ __forceinline__ Fixed fixed_point(double x, double scale) {
    const double r = rint(x * scale), hi = floor(r * (1.0 / 281474976710656.0));   // 2^48
    const double lo = fma(hi, -281474976710656.0, r) + 4503599627370496.0;         // in the low bits of 2^52 + lo
    Fixed f;
    f.w0 = (uint32_t)__double2loint(lo);
    f.w1 = (uint32_t)__double2hiint(lo) & 0xffffu;
    f.w2 = (uint32_t)__double2loint(hi + (4503599627370496.0 + 536870912.0));      // + 2^(kBias - 48)
    return f;
}
static_assert(kBias - kTop == 29, "bias of the top word");
// Whether that integer is the component itself (back = 1 / scale).
__device__ __forceinline__ bool held(double x, double scale, double back) { return rint(x * scale) * back == x; }

__device__ __forceinline__ bool refused(const ResPair& P) {
    return P.rounded[0] > P.limit[0] || P.rounded[1] > P.limit[1];
}

// Starts the counts of rounded components, and refuses a product whose operands
// are plainly not held: a cluster per operand takes 256 K of 64 rows and counts
// components that would be rounded even if the row's norm were the largest of
// them.  More than one in 512 (the limit is one in 2^15), and everything behind
// returns at once: a refused product costs 25 us more than the FP64 product
// alone, from 12% of it at the smallest size to 1% at chi = 1024.
constexpr int PROBE_C = 8, PROBE_T = 256, PROBE_K = 256;   // one row a warp
__global__ void __cluster_dims__(PROBE_C, 1, 1) __launch_bounds__(PROBE_T) res_probe_kernel(ResPair P) {
    __shared__ int total;
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    constexpr int ROWS = PROBE_C * PROBE_T / 32;
    const int w2 = blockIdx.x / PROBE_C, rank = blockIdx.x % PROBE_C, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const ResSource s = w2 ? P.s[1] : P.s[0];
    const cplx* x = row_ptr(s, (int)((long long)(rank * (PROBE_T / 32) + w) * s.rows / ROWS));
    cplx v[PROBE_K / 32];
    double mx = 0;
#pragma unroll
    for (int q = 0; q < PROBE_K / 32; ++q) v[q] = x[(long long)((q * 32 + lane) * s.K / PROBE_K) * s.sk];
    if (threadIdx.x == 0) total = 0;
    cluster.sync();
#pragma unroll
    for (int q = 0; q < PROBE_K / 32; ++q) mx = fmax(mx, fmax(fabs(v[q].x), fabs(v[q].y)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    int e = 0, lost = 0;
    frexp(mx, &e);
    e = min(kNormBits - e, 1000);
    const double scale = scalbn(1.0, e), back = scalbn(1.0, -e);
#pragma unroll
    for (int q = 0; q < PROBE_K / 32; ++q) lost += (held(v[q].x, scale, back) ? 0 : 1) + (held(v[q].y, scale, back) ? 0 : 1);
    lost = __reduce_add_sync(0xffffffffu, lost);
    if (lane == 0) atomicAdd(cluster.map_shared_rank(&total, 0), lost);
    cluster.sync();
    if (rank == 0 && threadIdx.x == 0)
        P.rounded[w2] = total > 2 * ROWS * PROBE_K / 512 && P.limit[w2] < kNormwise ? 1ull << 40 : 0ull;
}

// Per (K chunk, row): sum |x|^2 and max(|Re|, |Im|).  K contiguous: one block
// per row and chunk; else 32 rows per block, lanes along the rows.  The grid is
// what fits the chip (as in the kernels below): a refused product returns from
// a few blocks, not from tens of thousands.
__global__ void __launch_bounds__(NT) res_norm_kernel(ResPair P) {
    __shared__ double2 red[NT];
    if (refused(P)) return;
    const int items0 = P.nb[0] * P.nchunk[0], items = items0 + P.nb[1] * P.nchunk[1];
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int w2 = it >= items0 ? 1 : 0, q2 = it - (w2 ? items0 : 0);
        const ResSource s = w2 ? P.s[1] : P.s[0];
        const int nb = w2 ? P.nb[1] : P.nb[0], bx = q2 % nb, cy = q2 / nb;
        double2* part = w2 ? P.part[1] : P.part[0];
        const int chunk = w2 ? P.chunk[1] : P.chunk[0], k0 = cy * chunk, k1 = min(s.K, k0 + chunk);
        double sum = 0, mx = 0;
        auto take = [&](const cplx v) {
            sum = fma(v.x, v.x, fma(v.y, v.y, sum));     // a NaN survives here, fmax drops it
            mx = fmax(mx, fmax(fabs(v.x), fabs(v.y)));
        };
        __syncthreads();   // `red` of the item before has been read
        if (s.sk == 1) {
            const cplx* x = row_ptr(s, bx);
#pragma unroll 4
            for (int k = k0 + threadIdx.x; k < k1; k += NT) take(x[k]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                sum += __shfl_xor_sync(0xffffffffu, sum, o);
                mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            }
            if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = make_double2(sum, mx);
            __syncthreads();
            if (threadIdx.x == 0) {
                for (int q = 1; q < NT / 32; ++q) {
                    sum += red[q].x;
                    mx = fmax(mx, red[q].y);
                }
                part[(size_t)cy * s.rows + bx] = make_double2(sum, mx);
            }
        } else {
            const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
            const int row = bx * 32 + lane;
            if (row < s.rows) {
                const cplx* x = row_ptr(s, row);
#pragma unroll 4
                for (int k = k0 + w; k < k1; k += NT / 32) take(x[(long long)k * s.sk]);
            }
            red[threadIdx.x] = make_double2(sum, mx);
            __syncthreads();
            if (w == 0 && row < s.rows) {
                for (int q = 1; q < NT / 32; ++q) {
                    sum += red[q * 32 + lane].x;
                    mx = fmax(mx, red[q * 32 + lane].y);
                }
                part[(size_t)cy * s.rows + row] = make_double2(sum, mx);
            }
        }
    }
}

// Scale exponent e of each row (the row times 2^e has its 2-norm in
// (2^76, 2^77]), or kBadExp when an element is not finite.
__device__ __forceinline__ int row_exponent(const double2* __restrict__ part, int nchunk, int rows, int row, int K) {
    double sum = 0, mx = 0;
    for (int c = 0; c < nchunk; ++c) {
        const double2 v = part[(size_t)c * rows + row];
        sum += v.x;
        mx = fmax(mx, v.y);
    }
    if (isnan(sum) || isinf(mx)) return kBadExp;
    if (mx == 0.0) return 0;
    int e = 0;
    if (sum > 1e-270 && sum < 1e270) {
        frexp(sqrt(sum) * (1.0 + 1e-12), &e);                 // norm <= 2^e
    } else {                                                  // squares out of range: bound by the largest element
        frexp(mx, &e);
        int b = 0;
        frexp(sqrt(2.0 * K), &b);
        e += b;
    }
    return min(kNormBits - e, 1000);
}

// Residues of 16 rows x 128 K of an operand: planes[(3 l + c)][row][Kp] bytes,
// c = Re, Im, Re + Im.  Bound by instruction issue: 23 million complex
// elements (the operands of a chi=1024 Heisenberg product) write 1.4 GB, 0.21 ms
// at the HBM rate, take 0.48 ms and cost 20 x 20 integer instructions each.  A residue of
// the 78-bit integer is three dot products of its bytes with the powers of 2^8
// modulo p (dp4a), a quotient rounded in FP32 and one multiply-add.  A thread
// makes four consecutive K of a row at a time, so that a warp writes a whole
// 128-byte line of each plane.  The moduli are unrolled, so that their constants
// are immediates: read from constant memory in a loop they kept the address
// unit the busiest one.  A grid too small for the chip is split over the moduli
// as well.  A block that finds rounded components looks at the operand's count
// and leaves when it is past the limit, so that an operand for the FP64 product
// costs little here.
constexpr int CR = 16, CK = 128;
// kMagicI (1 - p) + the residue, which is in [0, p): t = 2^8 powers modulo p
// times the bytes, as the bits of a float; q = round((t - p/2) / p).
__device__ __forceinline__ uint32_t residue(const Fixed& v, uint32_t m0, uint32_t m1, uint32_t m2, uint32_t off, float inv,
                                            float half, uint32_t p) {
    const uint32_t t = __dp4a(v.w2, m2, __dp4a(v.w1, m1, __dp4a(v.w0, m0, off)));   // kMagicI + t, t < 2^20
    const float q = fmaf(__uint_as_float(t) - half, inv, kMagicF);
    return t - __float_as_uint(q) * p;
}
// The moduli L .. of [l0, l1) for four K of a row; their constants are immediates.
template <int L>
__device__ __forceinline__ void residues_of(const Fixed (&vr)[4], const Fixed (&vi)[4], uint8_t*& out, size_t plane, int l0,
                                            int l1) {
    if constexpr (L < NL) {
        if (L >= l0 && L < l1) {
            constexpr uint32_t p = kC.p[L], m0 = kC.m0[L], m1 = kC.m1[L], m2 = kC.m2[L], off = kC.off[L];
            constexpr float inv = kC.invf[L], half = kC.half[L];
            constexpr uint32_t twice = 2 * (kMagicI * (p - 1));
            uint32_t a[4], b[4], c[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                a[q] = residue(vr[q], m0, m1, m2, off, inv, half, p);
                b[q] = residue(vi[q], m0, m1, m2, off, inv, half, p);
                const uint32_t sum = a[q] + b[q] + twice;
                c[q] = min(sum, sum - p);   // the wrapped difference is large when sum < p
            }
            *reinterpret_cast<uint32_t*>(out) = pack4(a[0], a[1], a[2], a[3]);
            *reinterpret_cast<uint32_t*>(out + plane) = pack4(b[0], b[1], b[2], b[3]);
            *reinterpret_cast<uint32_t*>(out + 2 * plane) = pack4(c[0], c[1], c[2], c[3]);
            out += 3 * plane;
        }
        residues_of<L + 1>(vr, vi, out, plane, l0, l1);
    }
}

__global__ void __launch_bounds__(NT, 4) res_convert_kernel(ResPair P) {
    __shared__ cplx tile[CR][CK + 1];
    __shared__ double scale[CR], back[CR];
    __shared__ const cplx* rows[CR];
    if (__syncthreads_or(threadIdx.x == 0 && refused(P))) return;
    const int kb = (P.Kp + CK - 1) / CK, tid = threadIdx.x;
    const int w2 = (int)blockIdx.x >= P.nb[0] ? 1 : 0, bx = blockIdx.x - (w2 ? P.nb[0] : 0);
    const ResSource s = w2 ? P.s[1] : P.s[0];
    const int r0 = (bx / kb) * CR, k0 = (bx % kb) * CK;
    if (tid < CR) {
        const int row = r0 + tid;
        int e = 0;
        if (row < s.rows) {
            e = row_exponent(w2 ? P.part[1] : P.part[0], w2 ? P.nchunk[1] : P.nchunk[0], s.rows, row, s.K);
            if (k0 == 0 && blockIdx.y == 0) (w2 ? P.exps[1] : P.exps[0])[row] = e;
        }
        // a row that is not finite counts as 2^40 rounded components
        if (e == kBadExp && k0 == 0 && blockIdx.y == 0) atomicAdd(P.rounded + w2, 1ull << 40);
        scale[tid] = (e == kBadExp) ? 0.0 : scalbn(1.0, e);
        back[tid] = (e == kBadExp) ? 0.0 : scalbn(1.0, -e);
    } else if (tid >= 32 && tid < 32 + CR) {
        const int row = r0 + tid - 32;
        rows[tid - 32] = row < s.rows ? row_ptr(s, row) : nullptr;
    }
    __syncthreads();
    int lost = 0;   // rounded components among this thread's
    auto take = [&](int r, int k, const cplx v) {
        tile[r][k] = v;
        lost += (held(v.x, scale[r], back[r]) ? 0 : 1) + (held(v.y, scale[r], back[r]) ? 0 : 1);
    };
    if (s.sk == 1) {
#pragma unroll
        for (int i = 0; i < CR * CK / NT; ++i) {
            const int e = tid + i * NT, r = e / CK, k = e % CK;
            const cplx* x = rows[r];
            take(r, k, (x && k0 + k < s.K) ? x[k0 + k] : cmake(0, 0));
        }
    } else {
#pragma unroll
        for (int i = 0; i < CR * CK / NT; ++i) {
            const int e = tid + i * NT, r = e % CR, k = e / CR;
            const cplx* x = rows[r];
            take(r, k, (x && k0 + k < s.K) ? x[(k0 + k) * s.sk] : cmake(0, 0));
        }
    }
    bool past = false;
    if (lost > 0 && blockIdx.y == 0)
        past = atomicAdd(P.rounded + w2, (unsigned long long)lost) + lost > (w2 ? P.limit[1] : P.limit[0]);
    if (__syncthreads_or(past)) return;
    const size_t plane = (size_t)s.rows * P.Kp;
    const int l0 = blockIdx.y * P.lper, l1 = min(NL, l0 + P.lper), k = (tid & 31) * 4;
    for (int r = tid >> 5; r < CR; r += NT / 32) {
        const int row = r0 + r;
        if (row >= s.rows || k0 + k >= P.Kp) break;
        const double sc = scale[r];
        Fixed vr[4], vi[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            cplx v = tile[r][k + q];
            if (sc == 0.0) v = cmake(0, 0);
            vr[q] = fixed_point(v.x, sc);
            vi[q] = fixed_point(s.conj ? -v.y : v.y, sc);
        }
        uint8_t* out = (w2 ? P.planes[1] : P.planes[0]) + (size_t)row * P.Kp + k0 + k + (size_t)(3 * l0) * plane;
        residues_of<0>(vr, vi, out, plane, l0, l1);
    }
}

// ---- the GEMM ----------------------------------------------------------------------
constexpr int TM = 128, TN = 256, TKB = 128;   // tile rows, columns, K bytes per stage
constexpr int STAGES = 4;
constexpr int A_STAGE = TM * TKB, B_STAGE = TN * TKB;
constexpr int STAGE_BYTES = A_STAGE + B_STAGE;
constexpr int EPI_WARPS = 16, EPI_FIRST = 2;   // warps 0, 1: loads, MMAs
constexpr int EPI_COLS = 4 * TN / EPI_WARPS;   // columns per epilogue warp
constexpr int RG_THREADS = 32 * (EPI_FIRST + EPI_WARPS);
constexpr int TMEM_COLS = 512;
constexpr int CHUNK = 8;                        // columns per tensor-memory load
constexpr size_t RG_SMEM = (size_t)STAGES * STAGE_BYTES + 1024 + 256;

// kind::i8: D s32, A and B u8, both K-major, M x N.
constexpr uint32_t IDESC_I8 = (2u << 4) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);

__device__ __forceinline__ void mma_i8(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(IDESC_I8), "r"(accumulate)
        : "memory");
}

struct ResGemm {
    int M, N, nkb, mt, nt;   // K stages, row and column tiles
    int n4, mp;              // column groups of four and rows, padded to whole tiles
    uint32_t* res;           // [l][Re, Im][n4][mp] words of four columns
    ResidueGate gate;
    const DeviceWatch* watch;
};

// v modulo p in [0, p] (p itself for some multiples of p), |v| < 2^31: the
// quotient's error |v| / 2^39 stays below 1 / 256, so that flooring it is
// wrong at multiples of p only.
__device__ __forceinline__ uint32_t mod_int(int v, int p, int inv38) {
    return (uint32_t)(v - (__mulhi(v, inv38) >> 6) * p);
}

__device__ __forceinline__ void tmem_ldc(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__global__ void __launch_bounds__(RG_THREADS, 1)
residue_gemm_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, ResGemm P) {
    if (!residues_hold(P.gate)) return;
    extern __shared__ unsigned char rg_smem_raw[];
    const uint32_t raw = su32(rg_smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    const uint32_t bars = base + STAGES * STAGE_BYTES;
    const uint32_t full0 = bars, empty0 = bars + 8 * STAGES;
    const uint32_t accf0 = bars + 16 * STAGES, acce0 = accf0 + 16, drain = acce0 + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(rg_smem_raw + (drain + 8 - raw));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(accf0 + 8 * b, 1);
            mbar_init(acce0 + 8 * b, EPI_WARPS);
        }
        mbar_init(drain, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tmem_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_d = *tmem_slot;
    const int tiles = P.mt * P.nt, items = tiles * NL;

    if (warp == 0) {
        if (lane == 0) {
            const bool mute = blockIdx.x == 0 && (P.watch->mute >> WATCH_RESIDUE & 1u);
            int t = 0;
            bool ok = true;
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
                const int l = it / tiles, q = it % tiles, m0 = (q % P.mt) * TM, n0 = (q / P.mt) * TN;
                for (int c = 0; c < 3 && ok; ++c)
                    for (int kb = 0; kb < P.nkb; ++kb, ++t) {
                        const int s = t % STAGES;
                        if (!mbar_wait(empty0 + 8 * s, ((uint32_t)(t / STAGES) & 1u) ^ 1u, P.watch, WATCH_RESIDUE)) {
                            ok = false;
                            break;
                        }
                        if (t == 0 && mute) continue;   // test switch: this stage never arrives
                        mbar_expect_tx(full0 + 8 * s, STAGE_BYTES);
                        tma_load_3d(base + s * STAGE_BYTES, &mapA, kb * TKB, m0, 3 * l + c, full0 + 8 * s);
                        tma_load_3d(base + s * STAGE_BYTES + A_STAGE, &mapB, kb * TKB, n0, 3 * l + c, full0 + 8 * s);
                    }
            }
            if (!ok)   // an expired wait: the loads in flight land before the shared memory is given back
                for (int i = max(0, t - STAGES); i < t; ++i)
                    mbar_wait(full0 + 8 * (i % STAGES), (uint32_t)(i / STAGES) & 1u, P.watch, WATCH_RESIDUE);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            int t = 0, pass = 0;
            bool ok = true;
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x)
                for (int c = 0; c < 3 && ok; ++c, ++pass) {
                    const int b = pass & 1;
                    const uint32_t acc = tmem_d + (uint32_t)(b * TN);
                    if (!mbar_wait(acce0 + 8 * b, ((uint32_t)(pass >> 1) & 1u) ^ 1u, P.watch, WATCH_RESIDUE)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    for (int kb = 0; kb < P.nkb; ++kb, ++t) {
                        const int s = t % STAGES;
                        if (!mbar_wait(full0 + 8 * s, (uint32_t)(t / STAGES) & 1u, P.watch, WATCH_RESIDUE)) {
                            ok = false;
                            break;
                        }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint64_t da = smem_desc(base + s * STAGE_BYTES);
                        const uint64_t db = smem_desc(base + s * STAGE_BYTES + A_STAGE);
#pragma unroll
                        for (int ks = 0; ks < TKB / 32; ++ks)   // 32 bytes of K per instruction
                            mma_i8(acc, da + 2 * ks, db + 2 * ks, (kb | ks) ? 1u : 0u);
                        mma_commit(empty0 + 8 * s);
                    }
                    if (ok) mma_commit(accf0 + 8 * b);
                }
            if (!ok) {   // an expired wait: the MMAs issued end before the tensor memory is given back
                mma_commit(drain);
                mbar_wait(drain, 0, P.watch, WATCH_RESIDUE);
            }
        }
    } else if (warp >= EPI_FIRST) {
        // epilogue: warp w drains TMEM lanes 32*(w%4) .. +31 (a warp can reach
        // only those), columns [EPI_COLS h, EPI_COLS (h + 1)), h = (w-2)/4
        const int q = warp & 3, h = (warp - EPI_FIRST) >> 2;
        int pass = 0;
        bool ok = true;
        for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
            const int l = it / tiles, tq = it % tiles;
            const int m = (tq % P.mt) * TM + q * 32 + lane, n0 = (tq / P.mt) * TN + h * EPI_COLS;
            const int p = (int)kT.p[l], inv = kT.inv38[l];
            int acc[EPI_COLS];   // P1, then P1 + P2
#pragma unroll 1
            for (int c = 0; c < 3; ++c, ++pass) {
                const int b = pass & 1;
                ok = __all_sync(0xffffffffu, mbar_wait(accf0 + 8 * b, (uint32_t)(pass >> 1) & 1u, P.watch, WATCH_RESIDUE));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t src = tmem_d + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * TN + h * EPI_COLS);
                if (c == 0) {
#pragma unroll
                    for (int i = 0; i < EPI_COLS / CHUNK; ++i) {
                        uint32_t v[CHUNK];
                        tmem_ldc(src + CHUNK * i, v);
#pragma unroll
                        for (int e = 0; e < CHUNK; ++e) acc[CHUNK * i + e] = (int)v[e];
                    }
                } else {
                    // whole tiles are stored: res is padded to them
                    uint32_t* out = P.res + ((size_t)(2 * l + (c >> 1)) * P.n4 + n0 / 4) * P.mp + m;
                    const int sx = c == 1 ? -1 : 1;   // c = 1: P1 - P2; c = 2: P3 - (P1 + P2)
#pragma unroll
                    for (int i = 0; i < EPI_COLS / CHUNK; ++i) {
                        uint32_t v[CHUNK];
                        tmem_ldc(src + CHUNK * i, v);
#pragma unroll
                        for (int e = 0; e < CHUNK; e += 4) {
                            uint32_t r[4];
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                const int x = (int)v[e + u], y = acc[CHUNK * i + e + u];
                                r[u] = mod_int(sx * (x - y), p, inv);
                                acc[CHUNK * i + e + u] = y + x;
                            }
                            *out = pack4(r[0], r[1], r[2], r[3]);
                            out += P.mp;
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acce0 + 8 * b) : "memory");
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(TMEM_COLS)
                     : "memory");
    }
}

// ---- Chinese remainder theorem ---------------------------------------------------------
struct ResOut {
    cplx* C;
    int M, N, n4, mp, I;          // row m = (m % I) * 1 + (m / I) * sI
    long long sI, sn;
    const int *ea, *eb;       // scale exponents of A's rows and B's columns
    ResidueGate gate;
};

// The integer of C, rounded once to FP64.  S = sum_l r_l W_l as sh 2^115 +
// sm 2^75 + sl, sh and sm exact (sum r_l < 2^12.2, so sums below 2^52.7), sl
// to 2^39; the multiple of P removed; then h 2^40 + m as an unevaluated sum.
__device__ __forceinline__ double crt(const uint32_t (&w)[NL], int byte) {
    double sh = 0, sm = 0, sl = 0;
#pragma unroll
    for (int l = 0; l < NL; ++l) {
        const double d = __hiloint2double(0x43300000, __byte_perm(w[l], 0, 0x4440 | byte)) - 4503599627370496.0;
        sh = fma(d, kT.wh[l], sh);
        sm = fma(d, kT.wm[l], sm);
        sl = fma(d, kT.wl[l], sl);
    }
    const double k = rint(sh * (1.0 / kPh));
    const double h = fma(-k, kPh, sh) * 1099511627776.0;   // 2^40
    const double m = fma(-k, kPm, sm), l = fma(-k, kPl, sl);
    const double x = h + m, t = x - h, e = (h - (x - t)) + (m - t);
    constexpr double unit = 37778931862957161709568.0;     // 2^75
    return fma(x, unit, fma(e, unit, l));
}

__device__ __forceinline__ double pow2(int e) { return __hiloint2double((1023 + e) << 20, 0); }

__global__ void __launch_bounds__(128) res_crt_kernel(const uint32_t* __restrict__ res, ResOut o) {
    if (!residues_hold(o.gate)) return;
    const int m = blockIdx.x * 128 + threadIdx.x, g = blockIdx.y;
    if (m >= o.M) return;
    uint32_t wr[NL], wi[NL];
#pragma unroll
    for (int l = 0; l < NL; ++l) {
        wr[l] = res[((size_t)(2 * l) * o.n4 + g) * o.mp + m];
        wi[l] = res[((size_t)(2 * l + 1) * o.n4 + g) * o.mp + m];
    }
    const int ea = o.ea[m];
    cplx* row = o.C + (m % o.I) + (long long)(m / o.I) * o.sI;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int n = 4 * g + u;
        if (n >= o.N) break;
        const int eb = o.eb[n];
        // undo 2^(ea + eb) in three factors, so that no factor leaves FP64's range
        const int e = -(ea + eb), e1 = e / 3, e2 = (e - e1) / 2;
        const double f1 = pow2(e1), f2 = pow2(e2), f3 = pow2(e - e1 - e2);
        row[(long long)n * o.sn] = cmake(crt(wr, u) * f1 * f2 * f3, crt(wi, u) * f1 * f2 * f3);
    }
}

// rows x Kp int8, 3 NL planes
CUtensorMap make_map8(const uint8_t* ptr, int Kp, int rows, int rows_p, int box_rows) {
    CUtensorMap m;
    std::memset(&m, 0, sizeof(m));
    const cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)rows, (cuuint64_t)(3 * NL)};
    const cuuint64_t strides[2] = {(cuuint64_t)Kp, (cuuint64_t)Kp * rows_p};
    const cuuint32_t box[3] = {(cuuint32_t)TKB, (cuuint32_t)box_rows, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<uint8_t*>(ptr), dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        throw Error(NC_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
    return m;
}

int padded_k(int K) { return (K + 63) / 64 * 64; }
// Residue planes of both operands and the residues of C.
double scratch_bytes(long long M, long long N, long long K) {
    const double rows = (double)((M + TM - 1) / TM * TM), cols = (double)((N + TN - 1) / TN * TN);
    return 3.0 * NL * (double)(M + N) * padded_k((int)K) + 2.0 * NL * rows * cols;
}
constexpr double kMaxScratch = 16.0 * (1 << 30);

}  // namespace

// Measured on a B200, one H_eff product of a Heisenberg site (two GEMMs and
// the mix): the FP64 products alone / these, operands held / these, refused:
// chi = 256 146 / 183 / 196 us, 320 243 / 249 / 292, 384 330 / 298 / 376,
// 448 622 / 384 / 674, 512 869 / 452 / 921, 768 2301 / 945 / 2354,
// 1024 5718 / 1781 / 5781.  From 3 2^28 complex multiplications a GEMM (above
// chi = 384) a held product gains more than a refused one can lose; below one
// tile of rows or half a tile of columns the padding costs more.  Products
// whose residues would take more than 16 GB (several times the operands) or
// whose columns exceed the CRT's grid stay on the DMMA pipe.  Error against
// extended precision (2-norm, chi = 1024): DMMA 2.2e-15, this route 6.0e-17
// (one rounding; with 15 moduli 3.0e-16).
bool residue_gemm_pays(long long M, long long N, long long K) {
    return M >= TM && N >= TN / 2 && K >= 64 && K <= kMaxK && M * N * K >= (3LL << 28) && N <= 4 * 65535 &&
           scratch_bytes(M, N, K) <= kMaxScratch;
}

double residue_scratch_bytes(long long M, long long N, long long K) {
    return residue_gemm_pays(M, N, K) ? scratch_bytes(M, N, K) : 0;
}

namespace {

// Sizes of one product's launches, and its scratch: residue planes, row scales
// and partial norms of both operands, the counts of rounded components, and the
// residues of C.  One allocation, so that a product whose scratch cannot be had
// leaves nothing behind.
struct ResLayout {
    int Kp;
    int norm_blocks[2], nchunk[2], chunk[2];
    size_t planes[2], exps[2], part[2], rounded, res, bytes = 0;
    int mt, nt;
    size_t take(size_t n) {
        const size_t at = bytes;
        bytes += (n + 255) & ~size_t(255);
        return at;
    }
    ResLayout(const ResMatrix& a, const ResMatrix& b) {
        Kp = padded_k(a.K);
        const ResMatrix* const src[2] = {&a, &b};
        for (int w = 0; w < 2; ++w) {
            const ResMatrix& m = *src[w];
            // enough blocks for the chip: long K in chunks
            norm_blocks[w] = (m.sk == 1) ? m.rows : (m.rows + 31) / 32;
            const int want = std::max(1, std::min((4 * 148 + norm_blocks[w] - 1) / norm_blocks[w], (m.K + 63) / 64));
            chunk[w] = (m.K + want - 1) / want;
            nchunk[w] = (m.K + chunk[w] - 1) / chunk[w];
            planes[w] = take((size_t)3 * NL * m.rows * Kp);
            exps[w] = take(sizeof(int) * (size_t)m.rows);
            part[w] = take(sizeof(double2) * (size_t)nchunk[w] * m.rows);
        }
        rounded = take(2 * sizeof(unsigned long long));
        mt = (a.rows + TM - 1) / TM;
        nt = (b.rows + TN - 1) / TN;
        res = take(sizeof(uint32_t) * (size_t)2 * NL * (nt * (TN / 4)) * (mt * TM));
    }
};

// C(m,n) = sum_k A(m,k) B(n,k) to C[(m % I) + (m / I) * sI + n * sn] where the
// operands are held; the gate for the product that runs where they are not.
ResidueGate residue_product(Context& ctx, const ResMatrix& a, const ResMatrix& b, const ResLayout& lay, char* ws, cplx* C,
                            int I, long long sI, long long sn, bool normwise) {
    ResPair P;
    const ResMatrix* const src[2] = {&a, &b};
    ResidueGate gate;
    P.Kp = lay.Kp;
    P.rounded = reinterpret_cast<unsigned long long*>(ws + lay.rounded);
    gate.rounded = P.rounded;
    long long blocks = 0;
    int nb[2];
    for (int w = 0; w < 2; ++w) {
        const ResMatrix& m = *src[w];
        NC_ARG(m.rows >= 1 && m.K >= 1 && m.I >= 1 && (m.sk == 1 || m.si == 1), "residue operand: bad layout");
        ResSource& s = P.s[w];
        s.X = m.X; s.si = m.si; s.sI = m.sI; s.sk = m.sk; s.I = m.I; s.rows = m.rows; s.K = m.K; s.conj = m.conj;
        P.planes[w] = reinterpret_cast<uint8_t*>(ws + lay.planes[w]);
        P.exps[w] = reinterpret_cast<int*>(ws + lay.exps[w]);
        P.part[w] = reinterpret_cast<double2*>(ws + lay.part[w]);
        P.nb[w] = lay.norm_blocks[w]; P.chunk[w] = lay.chunk[w]; P.nchunk[w] = lay.nchunk[w];
        // random elements leave one component in 2^18 below 2^-24 of a norm (K = 1024); one graded K of a thousand leaves 2^-10
        P.limit[w] = normwise ? kNormwise : std::max(4ull, (unsigned long long)m.rows * m.K * 2 >> 15);
        gate.limit[w] = P.limit[w];
        const long long n = (long long)((P.Kp + CK - 1) / CK) * ((m.rows + CR - 1) / CR);
        nb[w] = (int)n;
        blocks += n;
    }
    NC_ARG(blocks < (1LL << 31), "residue operand: too large");
    res_probe_kernel<<<2 * PROBE_C, PROBE_T, 0, ctx.stream>>>(P);
    NC_CHECK_LAUNCH();
    const long long norms = (long long)P.nb[0] * P.nchunk[0] + (long long)P.nb[1] * P.nchunk[1];
    res_norm_kernel<<<(unsigned)std::min<long long>(norms, 148 * 8), NT, 0, ctx.stream>>>(P);
    NC_CHECK_LAUNCH();
    P.nb[0] = nb[0]; P.nb[1] = nb[1];
    P.lper = blocks < 2 * 148 ? 4 : blocks < 4 * 148 ? 7 : NL;
    res_convert_kernel<<<dim3((unsigned)blocks, (NL + P.lper - 1) / P.lper), NT, 0, ctx.stream>>>(P);
    NC_CHECK_LAUNCH();
    NC_SET_SMEM_ONCE(residue_gemm_kernel, RG_SMEM);
    ResGemm G;
    G.M = a.rows; G.N = b.rows;
    G.nkb = (lay.Kp + TKB - 1) / TKB;
    G.mt = lay.mt; G.nt = lay.nt;
    G.n4 = G.nt * (TN / 4);
    G.mp = G.mt * TM;
    G.res = reinterpret_cast<uint32_t*>(ws + lay.res);
    G.gate = gate;
    G.watch = ctx.watch;
    const CUtensorMap ma = make_map8(P.planes[0], lay.Kp, a.rows, a.rows, TM);
    const CUtensorMap mb = make_map8(P.planes[1], lay.Kp, b.rows, b.rows, TN);
    const long long items = (long long)G.mt * G.nt * NL;
    NC_ARG(items < (1LL << 31), "residue GEMM: too large");
    residue_gemm_kernel<<<(unsigned)std::min<long long>(items, 148), RG_THREADS, RG_SMEM, ctx.stream>>>(ma, mb, G);
    NC_CHECK_LAUNCH();
    ResOut o;
    o.C = C; o.M = G.M; o.N = G.N; o.n4 = G.n4; o.mp = G.mp; o.I = I; o.sI = sI; o.sn = sn;
    o.ea = P.exps[0]; o.eb = P.exps[1];
    o.gate = gate;
    const int groups = (G.N + 3) / 4;
    NC_ARG(groups <= 65535, "residue GEMM: too many columns");
    res_crt_kernel<<<dim3((G.M + 127) / 128, groups), 128, 0, ctx.stream>>>(G.res, o);
    NC_CHECK_LAUNCH();
    ctx.launches += 5;
    return gate;
}

}  // namespace

void zproduct(Context& ctx, const ZGemmParams& p, const ResMatrix& a, const ResMatrix& b, int I, long long sI,
              long long sn, bool normwise) {
    NC_ARG(a.K == b.K, "residue product: K");
    ArenaFrame f(ctx.scratch());
    if (!residue_gemm_pays(a.rows, b.rows, a.K)) {
        zgemm(p, ctx);
        return;
    }
    const ResLayout lay(a, b);
    if (!ctx.scratch().reserve(lay.bytes + zgemm_workspace_bytes(p) + 256)) {
        zgemm(p, ctx);   // the memory is taken: the product that needs (almost) none
        return;
    }
    profile_launch(ctx, 8.0 * a.rows * (double)b.rows * a.K, 0, [&] {
        ZGemmParams q = p;
        char* ws = ctx.scratch().alloc_n<char>(lay.bytes);
        q.gate = residue_product(ctx, a, b, lay, ws, p.C, I, sI, sn, normwise);
        zgemm_untimed(q, ctx);
    });
}

}  // namespace nc

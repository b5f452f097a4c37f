// mw_apply_fx.cu -- FP64-accuracy NS-form apply in 62-bit fixed point on the tensor cores.
//
// GB300's FP64 pipe runs 1.6 multiply-adds per SM and cycle, which bounds apply_kernel.  Here every
// operand of the three passes is a 62-bit fixed-point number with a power-of-two scale per row of an
// operator block and per column of the data, cut into seven signed 9-bit digits held as FP16
// integers.  A pass is a sum of 28 FP16 products (digit pairs i + j <= 6) on mma.sync.m16n8k16 with
// FP32 accumulation, and every sum is exact: see "ranges" below.  The dropped pairs (i + j >= 7) and
// the rounding of a pass's result to 62 bits are below 2^-58 of (row 1-norm) x (column maximum), less
// than FP64's own rounding of the same sums.
//
// Why mma.sync and not tcgen05: its accumulator fragment of one pass, once cut into digits, is the B
// fragment of the next (rows X' and columns Y of the x pass are columns X' and contraction index Y
// of the y pass), so the x and y passes run in a warp's registers.  With tcgen05 every intermediate
// would cross TMEM, registers and shared memory in 2-byte pieces; at these sizes that costs more
// than the tensor time it saves.  Bound: the mma.sync pipe (960 multiply-adds per SM and cycle, 600
// with the remainders of K = 9, 10), with the integer work of the digits close behind.
//
// Layout (one CTA per task, one warp per Z plane, for K > 8 per pair of planes):
//   x pass  T1[X'][Y, Z] = sum_X Ax[X'][X] in[X][Y, Z]     the warp's planes; data columns (Y, Z)
//   y pass  T2[Y'][X', Z] = sum_Y Ay[Y'][Y] T1[Y][X', Z]   the warp's planes; data columns X'
//   z pass  out[Z'][Y', X'] += sum_Z c Az[Z'][Z] T2[Z]     columns (Y', X') shared out among the warps
// T2 crosses the CTA through shared memory as digits, two Z to a word.  Rows of items as in
// apply_kernel: a row's x passes add up, its y and z passes run once.  Below the root scale the
// scaling-scaling path is left out exactly: u (wavelet-in-x part) comes from extra operator rows in
// the x pass's second row tile, and the (Y' < K, X' < K) columns of the z pass take a second operand
// whose Z < K part avoids that path.
//
// K > 8: the contraction index is 16 + (2K - 16).  The remainder's digit pairs are folded: one MMA
// carries four digit pairs of the same weight in its 16 k slots, 10 MMAs instead of 28.
//
// Ranges.  Operator rows are scaled by their 1-norm (sum_k |digit 0| <= 266), data columns by their
// maximum (|digit| <= 256), so a sum over one weight d = i + j is at most (number of pairs) x 20 x 2^16;
// the weights 4..6 are split over two accumulators, so that none exceeds 3 x 20 x 2^16 + 2^16 + ... <
// 2^22.  Accumulators start at 1.5 x 2^23, so every partial sum is an integer in [2^23, 2^24): exact in
// FP32, and the result's bits minus the start's are the integer.
#include "mw_chunks.cuh"
#include "mw_host.h"

#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

namespace mwg {

namespace {

constexpr int pitch_for(int cols) {  // columns padded so that four rows of eight words hit distinct banks
    int p = (cols + 7) / 8 * 8;
    while (p % 32 != 8 && p % 32 != 24) p += 8;
    return p;
}

template <int K>
struct FxGeo {
    static constexpr int N2 = 2 * K, NC = N2 * N2, K2 = K * K, K3 = K2 * K;
    static constexpr bool BIG = N2 > 16;              // contraction remainder and a second row tile
    static constexpr int PL = BIG ? 2 : 1;            // Z planes of a warp
    static constexpr int WARPS = N2 / PL, THREADS = 32 * WARPS;
    static constexpr int MINB = K == 4 ? 2 : 1;       // CTAs per SM that the registers are cut for
    static constexpr int UT = BIG ? 2 : 1;            // column tiles that have u
    static constexpr int RP = BIG ? 2 : 1;            // operator rows of a block per lane group of a warp (fx_rows)
    static constexpr int NT = (NC + 7) / 8;           // column tiles of the z pass
    static constexpr int NTX = (K2 + 7) / 8;          // ... of which take the second operand
    static constexpr int TPW = (NT + WARPS - 1) / WARPS;
    static constexpr int KE = (K + 1) / 2;            // Z pairs of the second operand
    static constexpr int P = pitch_for(NC), PE = pitch_for(K2);
    static constexpr int MAINW = 7 * 128;             // words of a row tile's digits (512 B per digit)
    static constexpr int TILEW = MAINW + (BIG ? 10 * 128 : 0);
    static constexpr int YT = BIG ? 2 : 1;            // row tiles of the y and z passes
    static constexpr int W_T2 = 7 * K * P, W_EX = 7 * KE * PE;
    static constexpr int O_EX = W_T2, O_X = O_EX + W_EX, O_Y = O_X + 4 * TILEW, O_Z = O_Y + YT * TILEW,
                         O_U = O_Z + YT * TILEW, WORDS = O_U + 2 * (PL * UT * 2) * THREADS;
    static_assert(W_T2 % 4 == 0 && W_EX % 4 == 0 && TILEW % 4 == 0, "16-byte aligned operator digits");
    static constexpr size_t SMEM = 4 * (size_t)WORDS;
    // input digits of a block: per warp and column tile (Y = 0..7, 8..15 of each plane; K > 8: 16.. of both)
    // the lanes' operands as 16-byte groups and one 8-byte group, then per warp the scale's exponent
    static constexpr int CT = N2 > 8 ? 2 : 1, TL = BIG ? 5 : CT, WB = BIG ? 18 : 14;
    static constexpr int IN_EXP = WARPS * TL * WB * 32, IN_WORDS = IN_EXP + 16;
};

constexpr float FX_MAGIC = 12582912.0f;  // 1.5 * 2^23
constexpr int FX_MAGIC_BITS = 0x4B400000;
constexpr int FX_SEG = 64;           // items whose pointers a CTA holds at a time
constexpr int FX_NONE = -1000000;  // exponent of a zero row or column

// accumulator of digit pair (i, d - i): weights 0..3 have one, 4..6 two
__device__ constexpr int fx_slot(int d, int i) { return d < 4 ? d : 4 + 2 * (d - 4) + ((i >= 2 && i <= 4) ? 1 : 0); }

// d (+)= a b; `first`: d starts at FX_MAGIC
__device__ __forceinline__ void fx_mma(float (&d)[4], const uint4 &a, uint32_t b0, uint32_t b1, bool first) {
    if (first) {
        const float c = FX_MAGIC;
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
            : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1), "f"(c));
    } else {
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
    }
}

// the data of one column tile: main digits (k = 2t, 2t+1 and 2t+8, 2t+9) and the folded remainder
struct FxB {
    uint32_t m[7][2];
    uint32_t s01, s23, s56, s4;
    // from this lane's pair of remainder elements (k = 16 + 2 (t & 1), + 1), up: t >= 2
    __device__ __forceinline__ void fold(const uint32_t (&q)[7], bool up) {
        s01 = up ? q[1] : q[0];
        s23 = up ? q[3] : q[2];
        s56 = up ? q[6] : q[5];
        s4 = up ? 0u : q[4];
    }
};

// D = operator digits (row tile at `frag`) x data digits, per weight
template <bool BIG>
__device__ __forceinline__ void fx_tile(float (&D)[10][4], const uint32_t *frag, const FxB &B, int lane) {
    const uint4 *f = reinterpret_cast<const uint4 *>(frag) + lane;
    if constexpr (BIG) {
        const uint4 *fr = f + 7 * 32;
#pragma unroll
        for (int d = 0; d < 4; d++) fx_mma(D[d], fr[d * 32], B.s01, B.s23, true);
#pragma unroll
        for (int d = 0; d < 3; d++) {
            fx_mma(D[4 + 2 * d], fr[(4 + 2 * d) * 32], B.s01, B.s56, true);
            fx_mma(D[5 + 2 * d], fr[(5 + 2 * d) * 32], B.s23, B.s4, true);
        }
    }
#pragma unroll
    for (int j = 0; j < 7; j++) {
        const uint4 a = f[j * 32];
#pragma unroll
        for (int i = 0; i < 7 - j; i++) {
            // an accumulator's first product in this order of (j, i) has the largest i
            const int d = i + j, imax = d < 4 ? d : (i >= 2 && i <= 4 ? 4 : (d == 4 ? 1 : d));
            fx_mma(D[fx_slot(d, i)], a, B.m[i][0], B.m[i][1], !BIG && i == imax);
        }
    }
}

// sum_d D_d 2^{9 (6 - d)} / 2^8 of register r: the pass's result in units of 2^-62 of its scale
__device__ __forceinline__ long long fx_value(const float (&D)[10][4], int r) {
    uint32_t I[10];  // the integers plus the accumulators' start; the starts are taken off in sums, modulo 2^32
#pragma unroll
    for (int a = 0; a < 10; a++) I[a] = __float_as_uint(D[a][r]);
    constexpr uint32_t M = FX_MAGIC_BITS;
    const uint32_t h = (I[0] << 9) + I[1];                                    // weights 0, 1: only the low 27 bits count
    const int m = (int)((I[2] << 9) + I[3] - (M * 513u));                     // weights 2, 3
    const int d4 = (int)(I[4] + I[5] - 2u * M);
    const int d6 = (int)(I[8] + I[9] + (128u - 2u * M));
    const int l = (int)(((I[6] + I[7]) << 1) + (uint32_t)(d6 >> 8) - 4u * M);  // weights 5, 6
    const long long v = (long long)d4 * 1024 + l + ((long long)m << 19);
    return (long long)((unsigned long long)v + ((unsigned long long)((h << 5) - (M * 513u << 5)) << 32));
}

// the seven digits of two 62-bit numbers as FP16 pairs (a in the low half)
__device__ __forceinline__ void fx_digits(long long a, long long b, uint32_t (&w)[7]) {
    constexpr unsigned long long BIAS = 256ull * (((1ull << 63) - 1) / 511ull);  // 256 in every digit
    const unsigned long long ua = (unsigned long long)a + BIAS, ub = (unsigned long long)b + BIAS;
    const __half2 off = __floats2half2_rn(1280.0f, 1280.0f);  // 1024 (the exponent pattern) + 256
#pragma unroll
    for (int s = 0; s < 7; s++) {
        const int sh = 9 * (6 - s);
        uint32_t x = (uint32_t)(ua >> sh), y = (uint32_t)(ub >> sh);
        uint32_t v = __byte_perm(x, y, 0x5410);
        v = s == 0 ? v : (v & 0x01ff01ffu);
        v |= 0x64006400u;
        __half2 h = __hsub2(*reinterpret_cast<__half2 *>(&v), off);
        w[s] = *reinterpret_cast<uint32_t *>(&h);
    }
}

// v 2^-right, rounded to nearest: a truncation here would be a bias that adds up over the items
__device__ __forceinline__ long long fx_shift(long long v, int right) {
    if (right <= 0) return (long long)((unsigned long long)v << min(-right, 63));
    return ((v >> min(right - 1, 62)) + 1) >> 1;
}

// the same with the two directions' counts and the rounding term prepared
struct FxShift {
    int left, right;
    long long half;
    __device__ __forceinline__ explicit FxShift(int d) : left(min(max(-d, 0), 63)), right(min(max(d, 0), 63)), half((1ll << right) >> 1) {}
    __device__ __forceinline__ long long operator()(long long v) const {
        return ((long long)((unsigned long long)v << left) + half) >> right;
    }
};

// f 2^e, rounded to nearest, without the FP64 pipe in the normal range
__device__ __forceinline__ double fx_to_double(long long f, int e) {
    const unsigned long long m = (unsigned long long)(f < 0 ? -f : f);
    const int lz = __clzll(m);
    const int ex = 63 - lz + e + 1023;  // exponent field
    if (m == 0 || ex < 1 || ex > 2046) return ldexp((double)f, e);
    const unsigned long long q = ((m << lz) + (1ull << 10)) >> 11;  // 53 bits; a carry out of rounding wraps m << lz
    const unsigned long long r = (m << lz) > 0xfffffffffffffbffull ? (1ull << 53) : q;
    return __longlong_as_double((long long)(((unsigned long long)(ex - 1) << 52) + r) | (f < 0 ? (long long)(1ull << 63) : 0));
}

// a double as a 62-bit fixed-point number of the scale 2^(efmax - 1022), efmax >= its exponent field
__device__ __forceinline__ long long fx_from_double(double x, int efmax) {
    const int hi = __double2hiint(x), lo = __double2loint(x);
    const int ef = (hi >> 20) & 0x7ff;
    const unsigned long long m = ((unsigned long long)((hi & 0xfffff) | 0x100000) << 32) | (unsigned)lo;
    const long long f = (long long)(((m << 10) >> min(efmax - ef, 63)) + 1) >> 1;
    return ef == 0 ? 0 : (hi < 0 ? -f : f);
}

// A 2K x 2K operator block's elements as a set of K warps holds them (unit = 0..K-1 the warp's place in
// the set): lane k of a row's lane group has element k of that row.  A warp takes two rows side by side
// where they fit (2K <= 16), else two one after the other.
template <int K>
__device__ __forceinline__ void fx_rows(double (&a)[FxGeo<K>::RP], const double *blk, int unit, int lane) {
    using G = FxGeo<K>;
    constexpr int LW = G::BIG ? 32 : 16;
    const int k = lane % LW;
#pragma unroll
    for (int i = 0; i < G::RP; i++) {
        const int r = G::BIG ? unit + i * K : 2 * unit + lane / LW;
        a[i] = k < G::N2 ? __ldg(blk + r * G::N2 + k) : 0.0;
    }
}

// These rows times cf into the digit fragments of the row tiles at d0 (rows 0..15) and d1 (rows 16.. as
// rows 4..; with U also u's rows, the wavelet columns of rows r < K: row 8 + r, or r - 8 for r >= 8, when
// K > 8, else row r), and the rows' exponents e: sum_k |a| <= 2^e.
template <int K, bool U>
__device__ __forceinline__ void fx_put(const double (&rows)[FxGeo<K>::RP], double cf, int unit, int lane, uint32_t *d0,
                                       uint32_t *d1, int *exps) {
    using G = FxGeo<K>;
    constexpr int LW = G::BIG ? 32 : 16;
    const int k = lane % LW;
    const unsigned mask = G::BIG ? 0xffffffffu : (lane < 16 ? 0xffffu : 0xffff0000u);
#pragma unroll
    for (int it = 0; it < G::RP; it++) {
        const int r = G::BIG ? unit + it * K : 2 * unit + lane / LW;
        const double a = rows[it] * cf;
        const int hi = __double2hiint(a), lo = __double2loint(a);
        const int ef = (hi >> 20) & 0x7ff;
        const int em = __reduce_max_sync(mask, ef);
        const unsigned m24 =
            ef == 0 ? 0u : ((((unsigned)((hi & 0xfffff) | 0x100000) << 3) | ((unsigned)lo >> 29)) >> min(em - ef, 31)) + 1u;
        const unsigned sum = __reduce_add_sync(mask, m24);
        const int e = em == 0 ? FX_NONE : 32 - __clz(sum) + em - 1046;
        const unsigned long long m = ((unsigned long long)((hi & 0xfffff) | 0x100000) << 32) | (unsigned)lo;
        const int sh = ef - 1013 - e;  // a 2^(62 - e) = mantissa 2^sh
        long long f = 0;
        if (ef != 0) f = (long long)(((sh >= -1 ? m << (sh + 1) : m >> min(-sh - 1, 63)) + 1) >> 1);
        if (hi < 0) f = -f;
        uint32_t q[7];
        fx_digits(f, 0, q);
        if (k == 0) exps[r] = e;
        if (k >= G::N2) continue;
#pragma unroll
        for (int u = 0; u < (U ? 2 : 1); u++) {
            const bool second = u || r >= 16;
            const int rr = u ? (G::BIG ? (r < 8 ? 8 + r : r - 8) : r) : (r >= 16 ? r - 12 : r);
            if (u && (r >= K || k < K)) continue;
            __half *base = reinterpret_cast<__half *>(second ? d1 : d0);
            if (k < 16) {
                __half *p = base + ((rr & 7) * 4 + ((k & 7) >> 1)) * 8 + ((rr >> 3) + 2 * (k >> 3)) * 2 + (k & 1);
#pragma unroll
                for (int j = 0; j < 7; j++) p[j * 256] = __ushort_as_half((unsigned short)q[j]);
            } else if constexpr (G::BIG) {
                const int kk = k - 16;
                __half *pr = base + 7 * 256;
#pragma unroll
                for (int f2 = 0; f2 < 10; f2++) {
                    const int d = f2 < 4 ? f2 : 4 + (f2 - 4) / 2;
#pragma unroll
                    for (int kap = 0; kap < 4; kap++) {
                        // the digit of the data in k group kap of this fragment's B operand
                        const int i = f2 < 4 ? kap : ((f2 & 1) ? kap + 2 : (kap < 2 ? kap : kap + 3));
                        if ((f2 >= 4 && (f2 & 1) && kap == 3) || d - i < 0 || d - i > 6) continue;
                        const int ks = 4 * kap + kk;
                        pr[f2 * 256 + ((rr & 7) * 4 + ((ks & 7) >> 1)) * 8 + ((rr >> 3) + 2 * (ks >> 3)) * 2 + (ks & 1)] =
                            __ushort_as_half((unsigned short)q[d - i]);
                    }
                }
            }
        }
    }
}

// The digits of input blocks as the x pass's column operands (FxGeo::IN_WORDS words per block): an input
// block serves a hundred items and more, so they are made once per apply.  One CTA per block, its warps
// as in the apply.
template <int K>
__global__ void __launch_bounds__(FxGeo<K>::THREADS) to_fx_kernel(const double *blocks, uint32_t *out, int nblocks) {
    using G = FxGeo<K>;
    constexpr int N2 = G::N2, K2 = G::K2, K3 = G::K3;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3, Z0 = G::PL * warp;
    for (int b = blockIdx.x; b < nblocks; b += gridDim.x) {
        const double *in = blocks + (size_t)b * 8 * K3;
        uint32_t *o = out + (size_t)b * G::IN_WORDS;
        int ef = 0;
        for (int i = lane; i < G::PL * G::NC; i += 32) {
            const int zi = i >= G::NC, q = i - zi * G::NC, c = q / K2, Z = Z0 + zi, cz = Z >= K;
            ef = max(ef, (__double2hiint(in[(size_t)(4 * cz + c) * K3 + (Z - cz * K) * K2 + (q - c * K2)]) >> 20) & 0x7ff);
        }
        ef = __reduce_max_sync(0xffffffffu, ef);
        if (lane == 0) o[G::IN_EXP + warp] = (uint32_t)(ef == 0 ? FX_NONE : ef - 1022);
        auto at = [&](int X, int Y, int Z) -> long long {
            if (X >= N2 || Y >= N2) return 0;
            const int cx = X >= K, cy = Y >= K, cz = Z >= K;
            return fx_from_double(
                in[(size_t)(cx + 2 * cy + 4 * cz) * K3 + (Z - cz * K) * K2 + (Y - cy * K) * K + (X - cx * K)], ef);
        };
        for (int ti = 0; ti < G::TL; ti++) {
            const bool rest = ti == G::PL * G::CT;  // K > 8: Y >= 16 of both planes
            const int zi = rest ? g >> 2 : ti / G::CT, Y = rest ? 16 + (g & 3) : 8 * (ti % G::CT) + g, Z = Z0 + zi;
            uint32_t w[G::WB];
            uint32_t q[7];
            fx_digits(at(2 * t, Y, Z), at(2 * t + 1, Y, Z), q);
#pragma unroll
            for (int s = 0; s < 7; s++) w[2 * s] = q[s];
            fx_digits(at(2 * t + 8, Y, Z), at(2 * t + 9, Y, Z), q);
#pragma unroll
            for (int s = 0; s < 7; s++) w[2 * s + 1] = q[s];
            if constexpr (G::BIG) {
                const int X = 16 + 2 * (t & 1);
                fx_digits(at(X, Y, Z), at(X + 1, Y, Z), q);
                FxB B;
                B.fold(q, t >= 2);
                w[14] = B.s01;
                w[15] = B.s23;
                w[16] = B.s56;
                w[17] = B.s4;
            }
            uint32_t *d = o + (warp * G::TL + ti) * G::WB * 32;
#pragma unroll
            for (int v = 0; v < G::WB / 4; v++)
                reinterpret_cast<uint4 *>(d)[v * 32 + lane] = make_uint4(w[4 * v], w[4 * v + 1], w[4 * v + 2], w[4 * v + 3]);
            reinterpret_cast<uint2 *>(d + (G::WB / 4) * 128)[lane] = make_uint2(w[G::WB - 2], w[G::WB - 1]);
        }
    }
}

// one lane's operand of column tile ti of a warp's planes
template <int K>
__device__ __forceinline__ void fx_load(FxB &B, const uint32_t *blk, int warp, int ti, int lane) {
    using G = FxGeo<K>;
    const uint32_t *d = blk + (warp * G::TL + ti) * G::WB * 32;
    uint32_t w[G::WB];
#pragma unroll
    for (int v = 0; v < G::WB / 4; v++) {
        const uint4 x = __ldg(reinterpret_cast<const uint4 *>(d) + v * 32 + lane);
        w[4 * v] = x.x;
        w[4 * v + 1] = x.y;
        w[4 * v + 2] = x.z;
        w[4 * v + 3] = x.w;
    }
    const uint2 y = __ldg(reinterpret_cast<const uint2 *>(d + (G::WB / 4) * 128) + lane);
    w[G::WB - 2] = y.x;
    w[G::WB - 1] = y.y;
#pragma unroll
    for (int s = 0; s < 7; s++) {
        B.m[s][0] = w[2 * s];
        B.m[s][1] = w[2 * s + 1];
    }
    if constexpr (G::BIG) {
        B.s01 = w[14];
        B.s23 = w[15];
        B.s56 = w[16];
        B.s4 = w[17];
    }
}

template <int K>
__global__ void __launch_bounds__(FxGeo<K>::THREADS, FxGeo<K>::MINB) apply_fx_kernel(ApplyLaunch L) {
    using G = FxGeo<K>;
    constexpr int N2 = G::N2, K2 = G::K2, K3 = G::K3;
    constexpr bool BIG = G::BIG;
    constexpr int YT = G::CT;              // column tiles of Y < 16 (K > 8: one more of Y >= 16 for both planes)
    constexpr int UT = G::UT, PL = G::PL;
    constexpr int RA = BIG ? 6 : 4;        // results of a thread per column tile
    extern __shared__ __align__(16) uint32_t fsm[];
    uint32_t *s_t2 = fsm, *s_ex = fsm + G::O_EX;
    long long *s_u = reinterpret_cast<long long *>(fsm + G::O_U) + threadIdx.x;  // u: a thread's own values
    __shared__ int s_node, s_redf;
    __shared__ int s_exx[2][32], s_exy[2][32], s_exz[2][32], s_e1[2][32];  // row exponents; T1's column exponents
    __shared__ const uint32_t *s_pi[FX_SEG];
    __shared__ const double *s_px[FX_SEG], *s_py[FX_SEG], *s_pz[FX_SEG];
    __shared__ double s_cf[FX_SEG];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const bool root = L.root != 0;
    const int Z0 = PL * warp;  // this warp's planes Z0 (and Z0 + 1)
    const bool ux[2] = {!root && Z0 < K, PL > 1 && !root && Z0 + 1 < K};  // the planes that have u
    // operator digits: sets of K warps; with twice as many warps the second set takes A_y and A_z
    const int unit = BIG || warp < K ? warp : warp - K;
    const bool put_x = BIG || warp < K, put_yz = BIG || warp >= K;

    for (int i = G::O_X + tid; i < G::WORDS; i += G::THREADS) fsm[i] = 0u;  // unused operator rows and columns
    if (tid < 64) (&s_exx[0][0])[tid] = (&s_exy[0][0])[tid] = (&s_exz[0][0])[tid] = FX_NONE;

    while (true) {
        __syncthreads();
        if (tid == 0) s_node = atomicAdd(L.counter, 1);
        if (tid < 64) (&s_e1[0][0])[tid] = FX_NONE;
        __syncthreads();
        const int w = s_node;
        if (w >= L.nnodes) break;
        const long long b0 = L.begin[w], b1 = L.end[w];
        // node accumulator: per column tile (8 nt + 2t, + 1) rows Z' = g, 8 + g, 12 + g (g >= 4), each
        // tile of a thread in units of 2^(ea - 62).  Indexed in a rolled loop, so it lives in local
        // memory between the z passes and leaves the registers to T1.
        long long acc[G::TPW][RA];
        int ea[G::TPW];
#pragma unroll 1
        for (int q = 0; q < G::TPW; q++) {
            ea[q] = 2 * FX_NONE;
            for (int r = 0; r < RA; r++) acc[q][r] = 0;
        }
        int nrows = 0, par = 0, xb = 0, zb = 0;
        const double *lastz = nullptr;
        for (long long sb = b0; sb < b1; sb += FX_SEG) {
            const int ni = (int)min((long long)FX_SEG, b1 - sb);
            if (sb != b0) __syncthreads();
            for (int i = tid; i < ni; i += G::THREADS) {
                s_pi[i] = reinterpret_cast<const uint32_t *>(L.in[sb + i]);
                s_px[i] = reinterpret_cast<const double *>(L.ax[sb + i]);
                s_py[i] = reinterpret_cast<const double *>(L.ay[sb + i]);
                s_pz[i] = reinterpret_cast<const double *>(L.az[sb + i]);
                s_cf[i] = L.coef[sb + i];
            }
            __syncthreads();
            double rx[G::RP], ry[G::RP], rz[G::RP];  // operator elements on their way
            if (put_x) fx_rows<K>(rx, s_px[0], unit, lane);
            if (put_yz) fx_rows<K>(ry, s_py[0], unit, lane);
            for (int j0 = 0; j0 < ni;) {
                int j1 = j0 + 1;  // the row: items of one term, ly and lz
                while (j1 < ni && s_py[j1] == s_py[j0] && s_pz[j1] == s_pz[j0]) j1++;
                const int hb = 32 - __clz(j1 - j0 - 1);  // head room of the row's sum, bits
                const bool single = j1 == j0 + 1, newz = s_pz[j0] != lastz;  // rows of one term and lz share A_z
                if (put_yz) fx_put<K, false>(ry, 1.0, unit, lane, fsm + G::O_Y, fsm + G::O_Y + G::TILEW, s_exy[par]);
                // T1: [plane][Y tile][register]; cm, cs: the tile Y >= 16 of both planes (K > 8)
                long long tm[PL][YT][4], ts[2][2][2], cm[4], cs[2];
                int et0 = FX_NONE, et1 = FX_NONE, et2 = FX_NONE;  // exponents of rows X' = g, 8 + g, 12 + g (u: 8 + g)
                for (int j = j0; j < j1; j++) {
                    const bool first = j == j0;
                    const uint32_t *in = s_pi[j];
                    FxB B, Bn;
                    fx_load<K>(Bn, in, warp, 0, lane);
                    const int ein = (int)__ldg(in + G::IN_EXP + warp);
                    uint32_t *fx0 = fsm + G::O_X + xb * 2 * G::TILEW, *fx1 = fx0 + G::TILEW;
                    if (put_x) fx_put<K, true>(rx, 1.0, unit, lane, fx0, fx1, s_exx[xb]);
                    __syncthreads();
                    if (put_x && j + 1 < ni) fx_rows<K>(rx, s_px[j + 1], unit, lane);
                    if (put_yz && first && newz) fx_rows<K>(rz, s_pz[j0], unit, lane);
                    const int ex0 = ein + s_exx[xb][g], ex1 = ein + s_exx[xb][8 + g],
                              ex2 = ein + s_exx[xb][g >= 4 ? 12 + g : 8 + g];
                    // sums of the row's items at a common exponent (hb bits of head room)
                    const int n0 = max(et0, ex0 + hb), n1 = max(et1, ex1 + hb), n2 = max(et2, ex2 + hb);
                    if (!first && __any_sync(0xffffffffu, n0 > et0 || n1 > et1 || n2 > et2)) {
                        // a larger scale than the row's so far: its sums move there
#pragma unroll
                        for (int zi = 0; zi < PL; zi++)
#pragma unroll
                            for (int tl = 0; tl < YT; tl++) {
#pragma unroll
                                for (int r = 0; r < 4; r++) tm[zi][tl][r] = fx_shift(tm[zi][tl][r], r < 2 ? n0 - et0 : n1 - et1);
#pragma unroll
                                for (int r = 0; r < 2; r++) {
                                    if constexpr (BIG) ts[zi][tl][r] = fx_shift(ts[zi][tl][r], n2 - et2);
                                    if (tl < UT && ux[zi]) {
                                        long long *u = s_u + ((zi * UT + tl) * 2 + r) * G::THREADS;
                                        *u = fx_shift(*u, n0 - et0);
                                    }
                                }
                            }
                        if constexpr (BIG) {
#pragma unroll
                            for (int r = 0; r < 4; r++) cm[r] = fx_shift(cm[r], r < 2 ? n0 - et0 : n1 - et1);
#pragma unroll
                            for (int r = 0; r < 2; r++) cs[r] = fx_shift(cs[r], n2 - et2);
                        }
                    }
                    // several items: every result moves right by at least the head room, rounded
                    const int m0 = min(n0 - ex0 - 1, 62), m1 = min(n1 - ex1 - 1, 62), m2 = min(n2 - ex2 - 1, 62);
                    auto add = [&](long long s, long long v, int m) -> long long {
                        if (single) return v;
                        v = ((v >> m) + 1) >> 1;
                        return first ? v : s + v;
                    };
                    float D[10][4];
#pragma unroll
                    for (int zi = 0; zi < PL; zi++) {
#pragma unroll
                        for (int tl = 0; tl < YT; tl++) {
                            B = Bn;  // the next tile's operand comes from L2 behind this one's products
                            if (zi * YT + tl + 1 < G::TL) fx_load<K>(Bn, in, warp, zi * YT + tl + 1, lane);
                            fx_tile<BIG>(D, fx0, B, lane);
#pragma unroll
                            for (int r = 0; r < 4; r++)
                                tm[zi][tl][r] = add(tm[zi][tl][r], fx_value(D, r), r < 2 ? m0 : m1);
                            if (BIG || (tl == 0 && ux[zi])) {
                                fx_tile<BIG>(D, fx1, B, lane);
#pragma unroll
                                for (int r = 0; r < 2; r++) {
                                    if constexpr (BIG) ts[zi][tl][r] = add(ts[zi][tl][r], fx_value(D, r), m2);
                                    if (ux[zi]) {
                                        long long *u = s_u + ((zi * UT + (BIG ? tl : 0)) * 2 + r) * G::THREADS;
                                        *u = add(*u, fx_value(D, (BIG ? 2 : 0) + r), m0);
                                    }
                                }
                            }
                        }
                    }
                    if constexpr (BIG) {
                        B = Bn;
                        fx_tile<BIG>(D, fx0, B, lane);
#pragma unroll
                        for (int r = 0; r < 4; r++) cm[r] = add(cm[r], fx_value(D, r), r < 2 ? m0 : m1);
                        fx_tile<BIG>(D, fx1, B, lane);
#pragma unroll
                        for (int r = 0; r < 2; r++) cs[r] = add(cs[r], fx_value(D, r), m2);
                    }
                    et0 = n0;
                    et1 = n1;
                    et2 = n2;
                    xb ^= 1;
                }
                // T1's columns to the largest magnitude over the CTA's planes
                {
                    auto mag = [](long long v) { return (unsigned long long)(v ^ (v >> 63)); };
                    unsigned long long o0 = 0, o1 = 0, o2 = 0;
#pragma unroll
                    for (int zi = 0; zi < PL; zi++)
#pragma unroll
                        for (int tl = 0; tl < YT; tl++) {
                            o0 |= mag(tm[zi][tl][0]) | mag(tm[zi][tl][1]);
                            o1 |= mag(tm[zi][tl][2]) | mag(tm[zi][tl][3]);
                            if constexpr (BIG) o2 |= mag(ts[zi][tl][0]) | mag(ts[zi][tl][1]);
                            if (tl < UT && ux[zi]) {
                                const long long *u = s_u + (zi * UT + tl) * 2 * G::THREADS;
                                o0 |= mag(u[0]) | mag(u[G::THREADS]);
                            }
                        }
                    if constexpr (BIG) {
                        o0 |= mag(cm[0]) | mag(cm[1]);
                        o1 |= mag(cm[2]) | mag(cm[3]);
                        o2 |= mag(cs[0]) | mag(cs[1]);
                    }
                    auto post = [&](unsigned long long o, int e, int X) {
                        o |= __shfl_xor_sync(0xffffffffu, o, 1);
                        o |= __shfl_xor_sync(0xffffffffu, o, 2);
                        if (t == 0 && o != 0 && X < N2) atomicMax(&s_e1[par][X], e + 2 - __clzll(o));  // |v| < 2^(64 - clz)
                    };
                    post(o0, et0, g);
                    if (N2 > 8) post(o1, et1, 8 + g);
                    if constexpr (BIG) post(o2, et2, g >= 4 ? 12 + g : 8 + (g & 1));
                }
                __syncthreads();
                if (newz) {
                    lastz = s_pz[j0];
                    zb ^= 1;
                    if (put_yz) fx_put<K, false>(rz, s_cf[j0], unit, lane, fsm + G::O_Z, fsm + G::O_Z + G::TILEW, s_exz[zb]);
                }
                if (put_yz && j1 < ni) fx_rows<K>(ry, s_py[j1], unit, lane);
                if (tid < 32) s_e1[par ^ 1][tid] = FX_NONE;
                // y pass, one column tile of X' at a time; results to shared memory as digits
                {
                    const FxShift d0(s_e1[par][g] - et0), d1(N2 > 8 ? s_e1[par][8 + g] - et1 : 0),
                        d2(BIG ? s_e1[par][g >= 4 ? 12 + g : 8 + (g & 1)] - et2 : 0);
                    const uint32_t *fy0 = fsm + G::O_Y, *fy1 = fy0 + G::TILEW;
                    // columns X' of tile kind 0: 0..7, 1: 8..15, 2: 16..19 (n >= 4) and u's 8, 9 (n < 2), 3: u's 0..7
                    auto run = [&](auto kind_c) {
                        constexpr int kind = decltype(kind_c)::value;
                        const FxShift &dk = kind == 1 ? d1 : (kind == 2 ? d2 : d0);
                        [[maybe_unused]] uint32_t wr[7];
                        if constexpr (BIG) {  // the remainder Y >= 16: lanes t < 2 hold plane 0, t >= 2 plane 1
                            const bool u8 = kind == 2 && g < 4;
                            const long long c0 = kind == 1 || u8 ? cm[2] : (kind == 2 ? cs[0] : cm[0]),
                                            c1 = kind == 1 || u8 ? cm[3] : (kind == 2 ? cs[1] : cm[1]);
                            const FxShift &dr = u8 ? d1 : dk;
                            fx_digits(dr(c0), dr(c1), wr);
                        }
#pragma unroll
                        for (int zi = 0; zi < PL; zi++) {
                            if (kind == 3 && !ux[zi]) continue;
                            const int Z = Z0 + zi;
                            FxB B;
                            uint32_t q[7];
                            long long p0, p1, p2 = 0, p3 = 0;  // Y = 2t, 2t + 1, 2t + 8, 2t + 9
                            if constexpr (kind == 0) {
                                p0 = tm[zi][0][0], p1 = tm[zi][0][1];
                                if constexpr (N2 > 8) p2 = tm[zi][YT - 1][0], p3 = tm[zi][YT - 1][1];
                            } else if constexpr (kind == 1) {
                                p0 = tm[zi][0][2], p1 = tm[zi][0][3];
                                p2 = tm[zi][YT - 1][2], p3 = tm[zi][YT - 1][3];
                            } else if constexpr (kind == 2) {
                                p0 = ts[zi][0][0], p1 = ts[zi][0][1];
                                p2 = g >= 4 || 8 + 2 * t < K ? ts[zi][1][0] : tm[zi][YT - 1][2];
                                p3 = g >= 4 || 9 + 2 * t < K ? ts[zi][1][1] : tm[zi][YT - 1][3];
                            } else {
                                const long long *u = s_u + zi * UT * 2 * G::THREADS;
                                p0 = 2 * t < K ? u[0] : tm[zi][0][0];
                                p1 = 2 * t + 1 < K ? u[G::THREADS] : tm[zi][0][1];
                                if constexpr (N2 > 8) {
                                    p2 = BIG && 8 + 2 * t < K ? u[2 * (UT - 1) * G::THREADS] : tm[zi][YT - 1][0];
                                    p3 = BIG && 9 + 2 * t < K ? u[(2 * (UT - 1) + 1) * G::THREADS] : tm[zi][YT - 1][1];
                                }
                            }
                            fx_digits(dk(p0), dk(p1), q);
#pragma unroll
                            for (int s = 0; s < 7; s++) B.m[s][0] = q[s];
                            if constexpr (N2 > 8) fx_digits(dk(p2), dk(p3), q);
#pragma unroll
                            for (int s = 0; s < 7; s++) B.m[s][1] = N2 > 8 ? q[s] : 0u;
                            if constexpr (BIG) {
                                const int src = 4 * g + (t & 1) + 2 * zi;
#pragma unroll
                                for (int s = 0; s < 7; s++) q[s] = __shfl_sync(0xffffffffu, wr[s], src);
                                B.fold(q, t >= 2);
                            }
                            // results of one row of Y' for columns n = 2t, 2t + 1: digit halves into the words of
                            // the plane's Z pair
                            auto put = [&](long long v0, long long v1, int Yq) {
                                fx_digits(v0, v1, q);
                                const int n = 2 * t;
                                const bool ext = kind == 3 || (kind == 2 && n < 2);
#pragma unroll
                                for (int b = 0; b < 2; b++) {
                                    const int nb = n + b;
                                    const int Xq = kind == 0 || kind == 3 ? nb : (kind == 1 || nb < 2 ? 8 + nb : (nb >= 4 ? 12 + nb : N2));
                                    unsigned short *o;
                                    int step;
                                    if (ext) {
                                        if (!ux[zi] || Yq >= K || Xq >= K) continue;
                                        o = reinterpret_cast<unsigned short *>(s_ex + (Z >> 1) * G::PE + Yq * K + Xq) + (Z & 1);
                                        step = 2 * G::KE * G::PE;
                                    } else {
                                        if (Yq >= N2 || Xq >= N2) continue;
                                        const int hy = Yq >= K, hx = Xq >= K;
                                        o = reinterpret_cast<unsigned short *>(
                                                s_t2 + (Z >> 1) * G::P + (2 * hy + hx) * K2 + (Yq - hy * K) * K + (Xq - hx * K)) + (Z & 1);
                                        step = 2 * K * G::P;
                                    }
#pragma unroll
                                    for (int s = 0; s < 7; s++) o[s * step] = (unsigned short)(b ? q[s] >> 16 : q[s]);
                                }
                            };
                            float D[10][4];
                            fx_tile<BIG>(D, fy0, B, lane);
                            put(fx_value(D, 0), fx_value(D, 1), g);
                            if constexpr (N2 > 8) put(fx_value(D, 2), fx_value(D, 3), 8 + g);
                            if constexpr (BIG && kind != 3) {
                                fx_tile<BIG>(D, fy1, B, lane);
                                put(fx_value(D, 0), fx_value(D, 1), g >= 4 ? 12 + g : N2);
                            }
                        }
                    };
                    run(std::integral_constant<int, 0>());
                    if constexpr (N2 > 8) run(std::integral_constant<int, 1>());
                    if constexpr (BIG) run(std::integral_constant<int, 2>());
                    if (ux[0]) run(std::integral_constant<int, 3>());
                }
                __syncthreads();
                // z pass over this warp's column tiles
                const uint32_t *fz0 = fsm + G::O_Z, *fz1 = fz0 + G::TILEW;
                const int ez0 = s_exz[zb][g], ez1 = s_exz[zb][8 + g], ez2 = s_exz[zb][g >= 4 ? 12 + g : 31];
#pragma unroll 1
                for (int q = 0; q < G::TPW; q++) {
                    const int nt = warp + q * G::WARPS;
                    if (nt >= G::NT) continue;
                    // word of Z pair zp, digit s, column 8 nt + g; second operand: Z < K from s_ex
                    auto word = [&](int s, int zp, bool second) -> uint32_t {
                        if (zp >= K) return 0u;
                        const int c = 8 * nt + g;
                        if (!second || zp >= G::KE) return s_t2[(s * K + zp) * G::P + c];
                        uint32_t e = s_ex[(s * G::KE + zp) * G::PE + c];
                        if ((K & 1) && zp == G::KE - 1) e = __byte_perm(e, s_t2[(s * K + zp) * G::P + c], 0x7610);
                        return e;
                    };
                    auto operand = [&](FxB &B, bool second) {
#pragma unroll
                        for (int s = 0; s < 7; s++) {
                            B.m[s][0] = word(s, t, second);
                            B.m[s][1] = word(s, t + 4, second);
                        }
                        if constexpr (BIG) {
                            const int zp = 8 + (t & 1), h = t >> 1;
                            B.s01 = word(h, zp, second);
                            B.s23 = word(2 + h, zp, second);
                            B.s56 = word(5 + h, zp, second);
                            B.s4 = h ? 0u : word(4, zp, second);
                        }
                    };
                    FxB B;
                    float D[10][4];
                    long long v[RA];
                    operand(B, false);
                    fx_tile<BIG>(D, fz0, B, lane);
#pragma unroll
                    for (int r = 0; r < 4; r++) v[r] = fx_value(D, r);
                    if constexpr (BIG) {
                        fx_tile<BIG>(D, fz1, B, lane);
#pragma unroll
                        for (int r = 0; r < 2; r++) v[4 + r] = fx_value(D, r);
                    }
                    if (!root && nt < G::NTX) {
                        operand(B, true);
                        fx_tile<BIG>(D, fz0, B, lane);
#pragma unroll
                        for (int r = 0; r < 4; r++) {
                            const int Zq = r < 2 ? g : 8 + g;
                            if (8 * nt + 2 * t + (r & 1) < K2 && Zq < K) v[r] = fx_value(D, r);
                        }
                    }
                    int ec[2];
#pragma unroll
                    for (int b = 0; b < 2; b++) {
                        const int c = min(8 * nt + 2 * t + b, G::NC - 1), hq = c / K2, rq = c - hq * K2, yq = rq / K;
                        ec[b] = s_e1[par][(hq & 1) * K + rq - yq * K] + s_exy[par][(hq >> 1) * K + yq];
                    }
                    int e[RA];
#pragma unroll
                    for (int r = 0; r < RA; r++) e[r] = ec[r & 1] + (r < 2 ? ez0 : (r < 4 ? ez1 : ez2));
                    int em = e[0];
#pragma unroll
                    for (int r = 1; r < RA; r++) em = max(em, e[r]);
                    long long s[RA];
                    int eq = ea[q];
                    const int up = max(em - eq, 0);
                    eq += up;
                    int over = 0;
#pragma unroll
                    for (int r = 0; r < RA; r++) {
                        const int sh = min(eq - e[r], 63);
                        s[r] = (up ? fx_shift(acc[q][r], up) : acc[q][r]) + ((v[r] + ((1ll << sh) >> 1)) >> sh);
                        const int hi = (int)(s[r] >> 32);
                        over |= hi ^ (hi >> 31);
                    }
                    const int room = (over >> 29) ? 2 : 0;  // |sum| >= 2^61: make room for the next row's 2^62
                    ea[q] = eq + room;
#pragma unroll
                    for (int r = 0; r < RA; r++) acc[q][r] = s[r] >> room;
                }
                nrows++;
                par ^= 1;
                j0 = j1;
            }
        }
        // a chunk's partial block is this task's alone; a whole node's block takes other tiers' sums too
        const bool set = L.set || (L.red_of && L.red_of[w] >= 0);
        double *out = L.out[w];
#pragma unroll 1
        for (int q = 0; q < G::TPW; q++) {
            const int nt = warp + q * G::WARPS;
            if (nt >= G::NT) continue;
#pragma unroll
            for (int r = 0; r < RA; r++) {
                const int c = 8 * nt + 2 * t + (r & 1), Zq = r < 2 ? g : (r < 4 ? 8 + g : (g >= 4 ? 12 + g : N2));
                if (c >= G::NC || Zq >= N2) continue;
                const int hq = c / K2, hz = Zq >= K;
                const double v = fx_to_double(acc[q][r], ea[q] - 62);
                double *o = out + (hq + 4 * hz) * K3 + (Zq - hz * K) * K2 + (c - hq * K2);
                *o = set ? v : *o + v;
            }
        }
        __syncthreads();
        if (tid == 0 && nrows > 0 && L.rows) atomicAdd(L.rows, nrows);
        finish_chunk(L, w, 8 * K3, &s_redf);
    }
}

template <int K>
void launch_fx(const ApplyLaunch &L, cudaStream_t s) {
    using G = FxGeo<K>;
    kernel_smem((const void *)apply_fx_kernel<K>, (int)G::SMEM);
    // one CTA per task (tasks are ordered longest first and taken in that order): CTAs end
    // throughout the launch, so kernels of other streams get SM slots without waiting for it
    apply_fx_kernel<K><<<L.nnodes, G::THREADS, G::SMEM, s>>>(L);
    MWG_CUDA(cudaGetLastError());
}

template <int K>
void launch_to_fx(const double *blocks, uint32_t *out, size_t n, cudaStream_t s) {
    to_fx_kernel<K><<<(int)std::min<size_t>(n, 65535), FxGeo<K>::THREADS, 0, s>>>(blocks, out, (int)n);
    MWG_CUDA(cudaGetLastError());
}

}  // namespace

size_t fx_words(int K) {
    switch (K) {
        case 4: return FxGeo<4>::IN_WORDS;
        case 5: return FxGeo<5>::IN_WORDS;
        case 6: return FxGeo<6>::IN_WORDS;
        case 7: return FxGeo<7>::IN_WORDS;
        case 8: return FxGeo<8>::IN_WORDS;
        case 9: return FxGeo<9>::IN_WORDS;
        case 10: return FxGeo<10>::IN_WORDS;
        default: throw Error(MW_ERR_ARG, "no fixed-point apply kernel for this order");
    }
}

void k_to_fx(const double *blocks, uint32_t *out, size_t n, int K, cudaStream_t s) {
    if (n == 0) return;
    switch (K) {
        case 4: launch_to_fx<4>(blocks, out, n, s); break;
        case 5: launch_to_fx<5>(blocks, out, n, s); break;
        case 6: launch_to_fx<6>(blocks, out, n, s); break;
        case 7: launch_to_fx<7>(blocks, out, n, s); break;
        case 8: launch_to_fx<8>(blocks, out, n, s); break;
        case 9: launch_to_fx<9>(blocks, out, n, s); break;
        case 10: launch_to_fx<10>(blocks, out, n, s); break;
        default: throw Error(MW_ERR_ARG, "no fixed-point apply kernel for this order");
    }
}

void k_apply_fx(const DevBasis &b, const ApplyLaunch &L, cudaStream_t s) {
    if (L.nnodes <= 0) return;
    switch (b.K) {
        case 4: launch_fx<4>(L, s); break;
        case 5: launch_fx<5>(L, s); break;
        case 6: launch_fx<6>(L, s); break;
        case 7: launch_fx<7>(L, s); break;
        case 8: launch_fx<8>(L, s); break;
        case 9: launch_fx<9>(L, s); break;
        case 10: launch_fx<10>(L, s); break;
        default: throw Error(MW_ERR_ARG, "no fixed-point apply kernel for this order");
    }
}

}  // namespace mwg

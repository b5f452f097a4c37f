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
// Why mma.sync and not tcgen05: an item needs ten accumulators (one per weight, two for the widest)
// and its digits cut anew before each pass, and that integer work takes about as long as the tensor
// pipe at mma.sync's rate (960 multiply-adds per SM and cycle, measured; 20 of 42 thousand SM cycles
// per item at 2K = 20).  mma.sync's accumulator fragments turn into 62-bit numbers in the registers that
// hold them; through TMEM every one of the ten would be read back by a second instruction stream.
// Bound: latency.  The products' pipe and the issue slots are each busy less than half of the time at four warps
// per scheduler (registers); the warps wait for fixed-latency results, barriers and the pipe in turn.
//
// Layout (one CTA per task, 7 to 16 warps that share out the column tiles of every pass):
//   x pass  T[Z][Y][X'] = sum_X Ax[X'][X] in[X][Y, Z]    input digits read as they lie in memory
//   y pass  T[Z][Y'][X'] = sum_Y Ay[Y'][Y] T[Z][Y][X']   in place: a warp owns its columns (X', Z)
//   z pass  out[Z'][Y', X'] += sum_Z c Az[Z'][Z] T[Z]    columns (Y', X')
// T is int64 in shared memory (64 KB at 2K = 20), its row pitches 2 modulo 4 so that the rows 2t apart of
// one operand fall into distinct banks.  Digits are made where they serve many times: an input block's
// once per call, an operator block's once per level (op_to_fx_kernel; the z pass's with its term's
// coefficient), both laid out as mma.sync operands, the operators' copied to shared memory by cp.async one
// pass ahead.  Rows of items as in apply_kernel: a row's x passes add up, its y and z passes run once.
// Below the root scale the scaling-scaling path is left out exactly: u (wavelet-in-x part) comes from extra
// operator rows in the x pass's second row tile, and the (Y' < K, X' < K) columns of the z pass take a
// second operand whose Z < K part avoids that path.
//
// Measured on a full chip, ns per item, apply_kernel's FP64 pipe first and then this kernel:
// 2K = 20: 653, 134;  2K = 18: 444, 119;  2K = 16: 256, 40;  2K = 12: 91, 33.  With T in registers and the
// operators' digits made per item 2K = 20 took 172 and 2K = 12 36; with a row tile of their own for rows
// 16.. 2K = 20 took 147 and 2K = 18 133.  Tier 3 of the 16-orbital Helmholtz batch (22 thousand items, alone
// on the chip): 5.3 ms with their digits, 6.9 ms with the double-FP32 kernel it had.
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
#include "mw_fx_round.h"
#include "mw_host.h"

#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

namespace mwg {

namespace {

constexpr int fx_pitch(int n) {  // n or a little more, 2 modulo 4: int64 rows 2t apart hit distinct banks
    while (n % 4 != 2) n++;
    return n;
}
// warps of a CTA: a divisor of the column tiles' number (50, 41, 32, 25, 18, 13, 8) with little left over, at
// most 16 (128 registers).  Two CTAs of 8 at 2K = 16: one's products run during the other's barriers (40 ns per item on a
// full chip against 46 with one of 16; the FP64 Poisson apply alike).  Not at 2K = 18, 20, where shared memory
// holds one CTA; 17 warps at 2K = 20 (no nearly empty last round) spill: 146 ns against 134.
constexpr int fx_warps(int K) { return K == 10 ? 16 : K == 9 ? 14 : K == 8 ? 8 : K == 7 ? 13 : K == 6 ? 9 : K == 5 ? 7 : 8; }

template <int K>
struct FxGeo {
    static constexpr int N2 = 2 * K, NC = N2 * N2, K2 = K * K, K3 = K2 * K;
    static constexpr bool BIG = N2 > 16;              // contraction remainder and a second row tile
    static constexpr int WARPS = fx_warps(K), THREADS = 32 * WARPS;
    static constexpr int MINB = K == 8 || K <= 6 ? 2 : 1;  // CTAs per SM that the registers are cut for
    // column tiles of the x pass: Y = 0..7, 8..15 of every plane Z; K > 8: Y >= 16 of two planes together
    static constexpr int CT = N2 > 8 ? 2 : 1, GRP = BIG ? K : N2, TL = BIG ? 5 : CT, NTIN = GRP * TL;
    static constexpr int NT = (NC + 7) / 8;           // column tiles of the y and z passes
    static constexpr int NTX = (K2 + 7) / 8;          // ... of which take the second operand
    static constexpr int TPW = (NT + WARPS - 1) / WARPS;
    // T[Z][Y][X'] and u[Z][Y][X'] (Z, Y, X' < K), 62-bit numbers
    static constexpr int PX = fx_pitch(N2), PZ = fx_pitch(N2 * PX), UX = fx_pitch(K), UZ = fx_pitch(K * UX);
    static constexpr int MAINW = 7 * 128;             // words of a row tile's digits (512 B per digit)
    static constexpr int TILEW = MAINW + (BIG ? 10 * 128 : 0);
    static constexpr int STACKW = BIG ? 14 * 128 : 0;  // words of the stacked rows 16.. (fx_stack)
    // an operator in the x pass: row tile 1 (u's rows and 16..), row tile 0, the stack; in the others without tile 1
    static constexpr int YW = TILEW + STACKW, XW = TILEW + YW;
    static constexpr int O_U = 2 * N2 * PZ, O_X = O_U + 2 * K * UZ + (2 * K * UZ) % 4, O_Y = O_X + 2 * XW,
                         O_Z = O_Y + YW, WORDS = O_Z + YW;
    static constexpr size_t SMEM = 4 * (size_t)WORDS;
    // input digits of a block: per column tile the lanes' operands as 16-byte groups and one 8-byte group, then
    // the tiles' exponents
    static constexpr int WB = BIG ? 18 : 14, IN_EXP = NTIN * WB * 32, IN_WORDS = IN_EXP + (NTIN + 7) / 8 * 4;
    // operator digits of a block: the x pass's (the y pass's from X_Y on) and the rows' exponents; then those
    // of the block times its term's coefficient (the z pass's)
    static constexpr int X_Y = TILEW, X_EXP = XW, Z_OFF = X_EXP + 16, Z_EXP = YW, OP_WORDS = Z_OFF + Z_EXP + 16;
    static_assert(Z_OFF == (BIG ? 2 * (7 + 10) + 14 : 2 * 7) * 128 + 16, "the same for all K of a kind");
    static_assert(O_U % 4 == 0 && O_X % 4 == 0 && TILEW % 4 == 0 && IN_WORDS % 4 == 0, "16-byte aligned copies");
};

constexpr float FX_MAGIC = 12582912.0f;  // 1.5 * 2^23
constexpr int FX_MAGIC_BITS = 0x4B400000;
constexpr int FX_SEG = 32;           // items whose pointers and exponents a CTA holds at a time
constexpr int FX_NONE = -20000;      // exponent of a zero row or block

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

// Rows 16.. of an operator, four at most, would fill a quarter of a row tile of their own: instead row 4a + r
// of these tiles holds row 16 + r for the weight d = a (D[0]) or 4 + a (D[1], D[2]), with the digit d - j that
// goes with the data's digit j.  Eleven products and three of the folded remainder in place of 38, and
// three accumulators in place of ten.  The weights 4..6 are split over D[1] and D[2]: at most 64 x 2^16 in each.
__device__ __forceinline__ void fx_stack(float (&D)[3][4], const uint32_t *frag, const FxB &B, int lane) {
    const uint4 *f = reinterpret_cast<const uint4 *>(frag) + lane;
    fx_mma(D[0], f[11 * 32], B.s01, B.s23, true);
    fx_mma(D[1], f[13 * 32], B.s4, B.s56, true);
    fx_mma(D[2], f[12 * 32], B.s01, B.s23, true);
#pragma unroll
    for (int j = 0; j < 7; j++) {
        if (j < 4) fx_mma(D[0], f[j * 32], B.m[j][0], B.m[j][1], false);
        fx_mma(D[j >= 2 && j <= 4 ? 2 : 1], f[(4 + j) * 32], B.m[j][0], B.m[j][1], false);
    }
}

// row 16 + (g & 3), column 2t + b, in every lane: this lane's weights (a = g >> 2 and a + 2) and its partner's
__device__ __forceinline__ long long fx_stack_value(const float (&D)[3][4], int b, int g) {
    const int n0 = __float_as_int(D[0][b]) - FX_MAGIC_BITS, n2 = __float_as_int(D[0][2 + b]) - FX_MAGIC_BITS;
    const int p0 = (int)(__float_as_uint(D[1][b]) + __float_as_uint(D[2][b]) - 2u * FX_MAGIC_BITS);
    const int p2 = (int)(__float_as_uint(D[1][2 + b]) + __float_as_uint(D[2][2 + b]) + (128u - 2u * FX_MAGIC_BITS));
    const unsigned long long q = ((unsigned long long)(long long)n0 << 18) + (unsigned long long)(long long)n2;
    const unsigned long long c = (unsigned long long)(long long)p0;
    unsigned long long v = (g & 4) ? (q << 19) + (c << 1) : (q << 28) + (c << 10);
    v += (unsigned long long)(long long)(p2 >> 8);
    return (long long)(v + __shfl_xor_sync(0xffffffffu, v, 16));
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

// v 2^-d rounded to nearest, with the two directions' counts and the rounding term of fx_round prepared
struct FxShift {
    int left, right;
    long long half;
    __device__ __forceinline__ explicit FxShift(int d) : left(min(max(-d, 0), 63)), right(min(max(d, 0), 62)), half((1ll << right) >> 1) {}
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

template <int K>
struct FxRows {
    static constexpr int N = FxGeo<K>::BIG ? 2 : 1;
};

// A 2K x 2K operator block's elements as a set of K warps holds them (unit = 0..K-1 the warp's place in
// the set): lane k of a row's lane group has element k of that row.  A warp takes two rows side by side
// where they fit (2K <= 16), else two one after the other.
template <int K>
__device__ __forceinline__ void fx_rows(double (&a)[FxRows<K>::N], const double *blk, int unit, int lane) {
    using G = FxGeo<K>;
    constexpr int LW = G::BIG ? 32 : 16;
    const int k = lane % LW;
#pragma unroll
    for (int i = 0; i < FxRows<K>::N; i++) {
        const int r = G::BIG ? unit + i * K : 2 * unit + lane / LW;
        a[i] = k < G::N2 ? __ldg(blk + r * G::N2 + k) : 0.0;
    }
}

// These rows times cf into the digit fragments of row tile 0 at d0 (rows 0..15), of the stack at st (rows
// 16..; fx_stack) and with U of row tile 1 at d1 (rows 16.. as rows 4.., and u's rows, the wavelet columns of rows
// r < K: row 8 + r, or r - 8 for r >= 8, when K > 8, else row r), and the rows' exponents e: sum_k |a| <= 2^e.
template <int K, bool U>
__device__ __forceinline__ void fx_put(const double (&rows)[FxRows<K>::N], double cf, int unit, int lane, uint32_t *d0,
                                       uint32_t *d1, uint32_t *st, short *exps) {
    using G = FxGeo<K>;
    constexpr int LW = G::BIG ? 32 : 16;
    const int k = lane % LW;
    const unsigned mask = G::BIG ? 0xffffffffu : (lane < 16 ? 0xffffu : 0xffff0000u);
#pragma unroll
    for (int it = 0; it < FxRows<K>::N; it++) {
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
        if (k == 0) exps[r] = (short)e;
        if (k >= G::N2) continue;
        if constexpr (G::BIG) {
            if (r >= 16) {
                __half *base = reinterpret_cast<__half *>(st);
                auto put = [&](int tile, int a, int ks, int i) {  // digit i in row 4a + r - 16, slot ks
                    const int R = 4 * a + r - 16;
                    base[tile * 256 + ((R & 7) * 4 + ((ks & 7) >> 1)) * 8 + ((R >> 3) + 2 * (ks >> 3)) * 2 + (ks & 1)] =
                        __ushort_as_half((unsigned short)q[i]);
                };
#pragma unroll
                for (int d = 0; d < 7; d++)  // its weight
#pragma unroll
                    for (int j = 0; j <= d; j++) {  // the data's digit
                        if (k < 16)
                            put((d < 4 ? 0 : 4) + j, d & 3, k, d - j);
                        else
                            put(d < 4 ? 11 : j < 4 ? 12 : 13, d & 3, 4 * (j < 4 ? j : j == 4 ? 0 : j - 3) + k - 16, d - j);
                    }
            }
        }
#pragma unroll
        for (int u = 0; u < (U ? 2 : 1); u++) {
            if (!U && r >= 16) continue;
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

// kernel arguments by value: nothing to upload
struct FxOpJobs {
    static constexpr int MAX = 16;
    FxOpJob job[MAX];
};
struct FxSets {
    static constexpr int MAX = 16;
    const double *in[MAX];
    uint32_t *out[MAX];
    long long first[MAX + 1];  // blocks of the sets before
    int n;
    const double *const *list;  // or (n = 1): these blocks
    const PairTask *pairs;  // or (n = 1): pairs' parents, or the cubes of their children's scaling parts (up)
    int up;
};

// Operator blocks' digits (FxGeo::OP_WORDS words per block), the blocks of one scale of the grid's y-th
// operator.  One CTA of K warps per block: the row tiles are put together in shared memory and leave in
// 16-byte pieces.
template <int K>
__global__ void __launch_bounds__(32 * K) op_to_fx_kernel(__grid_constant__ const FxOpJobs jobs) {
    using G = FxGeo<K>;
    extern __shared__ __align__(16) uint32_t fsm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const FxOpJob &J = jobs.job[blockIdx.y];
    for (int b = blockIdx.x; b < J.n; b += gridDim.x) {
        int t = 0, hi = J.op.T;  // the last term whose first block is at most b
        while (hi - t > 1) {
            const int m = (t + hi) / 2;
            if (J.op.first[m * J.op.S + J.s] <= b)
                t = m;
            else
                hi = m;
        }
        const int ts = t * J.op.S + J.s;
        const double *block = J.op.b64 + (size_t)(J.op.off[ts] + b - J.op.first[ts]) * G::NC;
        uint32_t *out = J.out + (size_t)b * G::OP_WORDS;
        double rows[FxRows<K>::N];
        fx_rows<K>(rows, block, warp, lane);
        for (int i = threadIdx.x; i < G::OP_WORDS; i += 32 * K) {
            const bool exps = (i >= G::X_EXP && i < G::Z_OFF) || i >= G::Z_OFF + G::Z_EXP;
            fsm[i] = exps ? 0x10001u * (uint32_t)(FX_NONE & 0xffff) : 0u;  // rows that there are not
        }
        __syncthreads();
        fx_put<K, true>(rows, 1.0, warp, lane, fsm + G::X_Y, fsm, fsm + G::X_Y + G::TILEW,
                        reinterpret_cast<short *>(fsm + G::X_EXP));
        uint32_t *z = fsm + G::Z_OFF;
        fx_put<K, false>(rows, J.op.c[t], warp, lane, z, nullptr, z + G::TILEW, reinterpret_cast<short *>(z + G::Z_EXP));
        __syncthreads();
        for (int i = threadIdx.x; i < G::OP_WORDS / 4; i += 32 * K)
            reinterpret_cast<uint4 *>(out)[i] = reinterpret_cast<const uint4 *>(fsm)[i];
        __syncthreads();
    }
}

// plane Z and row Y of column n of the x pass's tile ti of plane group gr
template <int K>
__device__ __forceinline__ void fx_in_column(int gr, int ti, int n, int &Y, int &Z) {
    using G = FxGeo<K>;
    if (G::BIG && ti == 4) {
        Y = 16 + (n & 3);
        Z = 2 * gr + (n >> 2);
    } else {
        Y = 8 * (ti % G::CT) + n;
        Z = G::BIG ? 2 * gr + ti / G::CT : gr;
    }
}

// The digits of input blocks as the x pass's column operands (FxGeo::IN_WORDS words per block), one scale
// per column tile (16-bit exponents), for the blocks of several trees at once.  One CTA per block, a warp
// per tile.
template <int K>
__global__ void __launch_bounds__(FxGeo<K>::THREADS) to_fx_kernel(__grid_constant__ const FxSets S) {
    using G = FxGeo<K>;
    constexpr int N2 = G::N2, K2 = G::K2, K3 = G::K3;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const size_t cs = (size_t)(S.pairs && S.up ? 8 : 1) * K3;  // distance of a block's components
    const long long nb = S.first[S.n];
    for (long long b = blockIdx.x; b < nb; b += gridDim.x) {
        int k = 0;
        while (b >= S.first[k + 1]) k++;
        const double *in = S.list    ? S.list[b]
                           : S.pairs ? (S.up ? S.pairs[b].child0 : S.pairs[b].parent)
                                     : S.in[k] + (size_t)(b - S.first[k]) * 8 * K3;
        uint32_t *o = S.out[k] + (size_t)(b - S.first[k]) * G::IN_WORDS;
        auto at = [&](int X, int Y, int Z) -> double {
            if (X >= N2 || Y >= N2) return 0.0;
            const int cx = X >= K, cy = Y >= K, cz = Z >= K;
            return in[(cx + 2 * cy + 4 * cz) * cs + (Z - cz * K) * K2 + (Y - cy * K) * K + (X - cx * K)];
        };
        for (int tile = warp; tile < G::NTIN; tile += G::WARPS) {
            int Y, Z;
            fx_in_column<K>(tile / G::TL, tile % G::TL, g, Y, Z);
            // this lane's X of the column, every X in one lane (those of the remainder in two)
            constexpr int NX = G::BIG ? 6 : (N2 > 8 ? 4 : 2);
            double x[NX];
#pragma unroll
            for (int j = 0; j < NX; j++) x[j] = at(j < 4 ? 2 * t + (j & 1) + 8 * (j >> 1) : 16 + 2 * (t & 1) + (j & 1), Y, Z);
            int ef = 0;
#pragma unroll
            for (int j = 0; j < NX; j++) ef = max(ef, (__double2hiint(x[j]) >> 20) & 0x7ff);
            ef = __reduce_max_sync(0xffffffffu, ef);
            if (lane == 0) reinterpret_cast<short *>(o + G::IN_EXP)[tile] = (short)(ef == 0 ? FX_NONE : ef - 1022);
            uint32_t w[G::WB];
            uint32_t q[7];
            fx_digits(fx_from_double(x[0], ef), fx_from_double(x[1], ef), q);
#pragma unroll
            for (int s = 0; s < 7; s++) {
                w[2 * s] = q[s];
                w[2 * s + 1] = 0u;
            }
            if constexpr (N2 > 8) {
                fx_digits(fx_from_double(x[2], ef), fx_from_double(x[3], ef), q);
#pragma unroll
                for (int s = 0; s < 7; s++) w[2 * s + 1] = q[s];
            }
            if constexpr (G::BIG) {
                fx_digits(fx_from_double(x[4], ef), fx_from_double(x[5], ef), q);
                FxB B;
                B.fold(q, t >= 2);
                w[14] = B.s01;
                w[15] = B.s23;
                w[16] = B.s56;
                w[17] = B.s4;
            }
            uint32_t *d = o + (size_t)tile * G::WB * 32;
#pragma unroll
            for (int v = 0; v < G::WB / 4; v++)
                reinterpret_cast<uint4 *>(d)[v * 32 + lane] = make_uint4(w[4 * v], w[4 * v + 1], w[4 * v + 2], w[4 * v + 3]);
            reinterpret_cast<uint2 *>(d + (G::WB / 4) * 128)[lane] = make_uint2(w[G::WB - 2], w[G::WB - 1]);
        }
    }
}

// one lane's operand of an x-pass tile
template <int K>
__device__ __forceinline__ void fx_load(FxB &B, const uint32_t *blk, int tile, int lane) {
    using G = FxGeo<K>;
    const uint32_t *d = blk + tile * G::WB * 32;
    // volatile: the loads stay where they are written, ahead of a barrier or of the tile before
    uint32_t w[G::WB];
#pragma unroll
    for (int v = 0; v < G::WB / 4; v++)
        asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(w[4 * v]), "=r"(w[4 * v + 1]), "=r"(w[4 * v + 2]), "=r"(w[4 * v + 3])
                     : "l"(reinterpret_cast<const uint4 *>(d) + v * 32 + lane));
    asm volatile("ld.global.nc.v2.u32 {%0,%1}, [%2];"
                 : "=r"(w[G::WB - 2]), "=r"(w[G::WB - 1])
                 : "l"(reinterpret_cast<const uint2 *>(d + (G::WB / 4) * 128) + lane));
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

// One lane's operand of a y- or z-pass tile: p(k) is the column's k-th value, zero for k >= 2K.
template <int K, typename F>
__device__ __forceinline__ void fx_operand(FxB &B, int t, F p) {
    using G = FxGeo<K>;
    uint32_t q[7];
    fx_digits(p(2 * t), p(2 * t + 1), q);
#pragma unroll
    for (int s = 0; s < 7; s++) B.m[s][0] = q[s];
    if constexpr (G::N2 > 8) {
        fx_digits(p(2 * t + 8), p(2 * t + 9), q);
#pragma unroll
        for (int s = 0; s < 7; s++) B.m[s][1] = q[s];
    } else {
#pragma unroll
        for (int s = 0; s < 7; s++) B.m[s][1] = 0u;
    }
    if constexpr (G::BIG) {
        const int k = 16 + 2 * (t & 1);
        fx_digits(p(k), p(k + 1), q);
        B.fold(q, t >= 2);
    }
}

// column c of the y pass (a = Z) or z pass (a = Y'): the scaling columns (a < K, X' < K) first
template <int K>
__device__ __forceinline__ void fx_column(int c, int &a, int &x) {
    constexpr int K2 = K * K;
    const int q = c / K2, r = c - q * K2, i = r / K;
    a = (q >> 1) * K + i;
    x = (q & 1) * K + r - i * K;
}

__device__ __forceinline__ void fx_copy(uint32_t *dst, const uint32_t *src, int words) {
    for (int i = 4 * threadIdx.x; i < words; i += 4 * blockDim.x)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + i)),
                     "l"(src + i)
                     : "memory");
}

// every copy issued so far has landed, for all threads of the CTA
__device__ __forceinline__ void fx_landed() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
}

template <int K>
__global__ void __launch_bounds__(FxGeo<K>::THREADS, FxGeo<K>::MINB) apply_fx_kernel(ApplyLaunch L) {
    using G = FxGeo<K>;
    constexpr int N2 = G::N2, K2 = G::K2, K3 = G::K3, PX = G::PX, PZ = G::PZ, UX = G::UX, UZ = G::UZ;
    constexpr bool BIG = G::BIG;
    constexpr int RA = BIG ? 6 : 4;  // results of a thread per column tile
    extern __shared__ __align__(16) uint32_t fsm[];
    long long *s_t = reinterpret_cast<long long *>(fsm), *s_u = reinterpret_cast<long long *>(fsm + G::O_U);
    __shared__ int s_node, s_redf, s_e1[2][32];  // s_e1: T1's column exponents
    __shared__ const uint32_t *s_pi[FX_SEG], *s_px[FX_SEG], *s_py[FX_SEG], *s_pz[FX_SEG];
    __shared__ short s_ein[FX_SEG][(G::NTIN + 7) / 8 * 8];  // column exponents, per x-pass tile
    __shared__ short s_exx[FX_SEG][32], s_exy[FX_SEG][32], s_exz[FX_SEG][32];  // row exponents
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const bool root = L.root != 0;
    // the rows of this lane's results: g, 8 + g and, in the second row tile, 12 + g (g >= 4) or u's 8 + g
    const int x2 = g >= 4 ? 12 + g : 8 + g;

    while (true) {
        __syncthreads();
        if (tid == 0) s_node = atomicAdd(L.counter, 1);
        if (tid < 64) (&s_e1[0][0])[tid] = FX_NONE;
        __syncthreads();
        const int w = s_node;
        if (w >= L.nnodes) break;
        const long long b0 = L.begin[w], b1 = L.end[w];
        // node accumulator: per column tile of this warp (columns 8 nt + 2t, + 1) rows Z' = g, 8 + g, 12 + g
        // (g >= 4), each tile of a thread in units of 2^(ea - 62).  Indexed in a rolled loop, so it lives in
        // local memory between the z passes.
        long long acc[G::TPW][RA];
        int ea[G::TPW];
#pragma unroll 1
        for (int q = 0; q < G::TPW; q++) {
            ea[q] = -1000000;
            for (int r = 0; r < RA; r++) acc[q][r] = 0;
        }
        int nrows = 0, par = 0;
        for (long long sb = b0; sb < b1; sb += FX_SEG) {
            const int ni = (int)min((long long)FX_SEG, b1 - sb);
            if (sb != b0) __syncthreads();
            for (int i = tid; i < ni; i += G::THREADS) {
                s_pi[i] = reinterpret_cast<const uint32_t *>(L.in[sb + i]);
                s_px[i] = reinterpret_cast<const uint32_t *>(L.ax[sb + i]);
                s_py[i] = reinterpret_cast<const uint32_t *>(L.ay[sb + i]);
                s_pz[i] = reinterpret_cast<const uint32_t *>(L.az[sb + i]);
            }
            __syncthreads();
            fx_copy(fsm + G::O_X, s_px[0], G::XW);
            fx_copy(fsm + G::O_Y, s_py[0] + G::X_Y, G::YW);
            for (int i = tid; i < 32 * ni; i += G::THREADS) {
                const int j = i >> 5, r = i & 31;
                s_exx[j][r] = reinterpret_cast<const short *>(s_px[j] + G::X_EXP)[r];
                s_exy[j][r] = reinterpret_cast<const short *>(s_py[j] + G::X_EXP)[r];
                s_exz[j][r] = reinterpret_cast<const short *>(s_pz[j] + G::Z_EXP)[r];
            }
            for (int i = tid; i < ni * G::NTIN; i += G::THREADS) {
                const int j = i / G::NTIN, r = i - j * G::NTIN;
                s_ein[j][r] = reinterpret_cast<const short *>(s_pi[j] + G::IN_EXP)[r];
            }
            const uint32_t *lastz = nullptr;
            for (int j0 = 0; j0 < ni;) {
                int j1 = j0 + 1;  // the row: items of one term, ly and lz
                while (j1 < ni && s_py[j1] == s_py[j0] && s_pz[j1] == s_pz[j0]) j1++;
                const int hb = 32 - __clz(j1 - j0 - 1);  // head room of the row's sum, bits
                const bool single = j1 == j0 + 1;
                int h0 = 5 * FX_NONE, h1 = h0, h2 = h0;  // largest exponents of T1's rows X' = g, 8 + g, x2
                for (int j = j0; j < j1; j++) {
                    const bool first = j == j0, last = j + 1 == j1;
                    const uint32_t *in = s_pi[j];
                    FxB B, Bn;
                    if (warp < G::NTIN) fx_load<K>(Bn, in, warp, lane);
                    fx_landed();  // A_x (and A_y); the z pass has read T
                    if (first) {
                        if (s_pz[j0] != lastz) {  // rows of one term and lz share A_z
                            lastz = s_pz[j0];
                            fx_copy(fsm + G::O_Z, lastz, G::YW);
                        }
                    }
                    const int exg = s_exx[j][g], exh = s_exx[j][8 + g], exq = s_exx[j][x2];
                    const uint32_t *fx1 = fsm + G::O_X + (j & 1) * G::XW, *fx0 = fx1 + G::X_Y, *fxs = fx0 + G::TILEW;
                    if (j + 1 < ni) fx_copy(fsm + G::O_X + ((j + 1) & 1) * G::XW, s_px[j + 1], G::XW);
#pragma unroll 1
                    for (int tile = warp; tile < G::NTIN; tile += G::WARPS) {
                        B = Bn;  // the next tile's operand comes from L2 behind this one's products
                        if (tile + G::WARPS < G::NTIN) fx_load<K>(Bn, in, tile + G::WARPS, lane);
                        const int gr = tile / G::TL, ti = tile - gr * G::TL;
                        // the row's sums at the tile's largest exponents, with head room; of several items every
                        // result moves right by at least that, rounded
                        const int ej = s_ein[j][tile];
                        int et0 = ej + exg, et1 = ej + exh, et2 = ej + exq, m0 = 0, m1 = 0, m2 = 0;
                        if (!single) {
                            const int f0 = et0, f1 = et1, f2 = et2;
                            for (int i = j0; i < j1; i++) {
                                const int e = s_ein[i][tile];
                                et0 = max(et0, e + s_exx[i][g]);
                                et1 = max(et1, e + s_exx[i][8 + g]);
                                if (BIG) et2 = max(et2, e + s_exx[i][x2]);
                            }
                            et0 += hb;
                            et1 += hb;
                            et2 += hb;
                            m0 = min(et0 - f0 - 1, 62), m1 = min(et1 - f1 - 1, 62), m2 = min(et2 - f2 - 1, 62);
                        }
                        unsigned long long o0 = 0, o1 = 0, o2 = 0;
                        auto add = [&](long long *s, long long v, int m, unsigned long long &o) {
                            if (!single) {
                                v = ((v >> m) + 1) >> 1;
                                if (!first) v += *s;
                            }
                            *s = v;
                            o |= (unsigned long long)(v ^ (v >> 63));
                        };
                        int Y, Z;  // of column 2t; column 2t + 1 is Y + 1
                        fx_in_column<K>(gr, ti, 2 * t, Y, Z);
                        long long *T = s_t + Z * PZ + Y * PX, *u = s_u + Z * UZ + Y * UX;
                        float D[10][4];
                        fx_tile<BIG>(D, fx0, B, lane);
#pragma unroll
                        for (int r = 0; r < 4; r++)
                            if (g + 8 * (r >> 1) < N2 && Y + (r & 1) < N2)
                                add(T + (r & 1) * PX + g + 8 * (r >> 1), fx_value(D, r), r < 2 ? m0 : m1, r < 2 ? o0 : o1);
                        const bool has_u = !root && Z < K && Y < K;
                        if (BIG && (root || ti == 4 || 2 * gr + ti / 2 >= K)) {  // no column with u (the warp's tile as a whole)
                            float E[3][4];
                            fx_stack(E, fxs, B, lane);
#pragma unroll
                            for (int r = 0; r < 2; r++) {
                                const long long v = fx_stack_value(E, r, g);
                                if (g >= 4 && 12 + g < N2 && Y + r < N2) add(T + r * PX + 12 + g, v, m2, o2);
                            }
                        } else if constexpr (BIG) {
                            fx_tile<BIG>(D, fx1, B, lane);
#pragma unroll
                            for (int r = 0; r < 2; r++) {
                                if (g >= 4 && 12 + g < N2 && Y + r < N2) add(T + r * PX + 12 + g, fx_value(D, r), m2, o2);
                                if (g < 2 && 8 + g < K && has_u && Y + r < K) add(u + r * UX + 8 + g, fx_value(D, r), m2, o2);
                                if (has_u && Y + r < K) add(u + r * UX + g, fx_value(D, 2 + r), m0, o0);
                            }
                        } else if (!root && ti == 0 && gr < K) {
                            fx_tile<BIG>(D, fx1, B, lane);
#pragma unroll
                            for (int r = 0; r < 2; r++)
                                if (g < K && Y + r < K) add(u + r * UX + g, fx_value(D, r), m0, o0);
                        }
                        if (last) {  // |v| < 2^(64 - clz)
                            if (o0) h0 = max(h0, et0 + 2 - __clzll(o0));
                            if (o1) h1 = max(h1, et1 + 2 - __clzll(o1));
                            if (o2) h2 = max(h2, et2 + 2 - __clzll(o2));
                        }
                    }
                }
                // T1's columns X' to their largest magnitude
                {
                    auto post = [&](int e, int X) {
                        e = max(e, __shfl_xor_sync(0xffffffffu, e, 1));
                        e = max(e, __shfl_xor_sync(0xffffffffu, e, 2));
                        if (t == 0 && e > FX_NONE) atomicMax(&s_e1[par][X], e);
                    };
                    post(h0, g);
                    if (N2 > 8) post(h1, 8 + g);
                    if constexpr (BIG) post(h2, x2);
                }
                fx_landed();
                if (tid < 32) s_e1[par ^ 1][tid] = FX_NONE;
                // y pass in place: a warp reads its 8 columns (Z, X') whole before it writes them
                const uint32_t *fy0 = fsm + G::O_Y, *fys = fy0 + G::TILEW;
#pragma unroll 1
                for (int tile = warp; tile < G::NT; tile += G::WARPS) {
                    const int c = 8 * tile + g;
                    int Z, X;
                    fx_column<K>(min(c, G::NC - 1), Z, X);
                    // T1's exponents by the x-pass tiles that Y = 0..7, 8..15 and 16.. came from
                    const int gr = BIG ? Z >> 1 : Z, it = gr * G::TL + (BIG ? (Z & 1) * G::CT : 0);
                    int e0 = 5 * FX_NONE, e1 = e0, e2 = e0;
                    for (int i = j0; i < j1; i++) {
                        const int ex = s_exx[i][X] + hb;
                        e0 = max(e0, s_ein[i][it] + ex);
                        if (N2 > 8) e1 = max(e1, s_ein[i][it + 1] + ex);
                        if (BIG) e2 = max(e2, s_ein[i][gr * G::TL + 4] + ex);
                    }
                    const int ee = s_e1[par][X];
                    const FxShift sh0(ee - e0), sh1(ee - e1), sh2(ee - e2);
                    auto sh = [&](long long v, int Y) { return Y < 8 ? sh0(v) : (Y < 16 ? sh1(v) : sh2(v)); };
                    const long long *T = s_t + Z * PZ + X, *u = s_u + Z * UZ + X;
                    int Zr[2], Xr[2];  // of the results' columns 2t, 2t + 1
#pragma unroll
                    for (int b = 0; b < 2; b++) fx_column<K>(min(8 * tile + 2 * t + b, G::NC - 1), Zr[b], Xr[b]);
                    FxB B;
                    float D[10][4];
                    if (!root && tile < G::NTX) {  // scaling columns: u where Y < K
                        const bool in = c < K2;
                        fx_operand<K>(B, t, [&](int Y) -> long long {
                            return !in || Y >= N2 ? 0 : sh(Y < K ? u[Y * UX] : T[Y * PX], Y);
                        });
                        fx_tile<BIG>(D, fy0, B, lane);
                        __syncwarp();
#pragma unroll
                        for (int r = 0; r < 4; r++) {
                            const int Yq = g + 8 * (r >> 1), b = r & 1;
                            if (Yq < K && 8 * tile + 2 * t + b < K2) s_u[Zr[b] * UZ + Yq * UX + Xr[b]] = fx_value(D, r);
                        }
                    }
                    const bool in = c < G::NC;
                    fx_operand<K>(B, t, [&](int Y) -> long long { return !in || Y >= N2 ? 0 : sh(T[Y * PX], Y); });
                    fx_tile<BIG>(D, fy0, B, lane);
                    __syncwarp();
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const int Yq = g + 8 * (r >> 1), b = r & 1;
                        if (Yq < N2 && 8 * tile + 2 * t + b < G::NC) s_t[Zr[b] * PZ + Yq * PX + Xr[b]] = fx_value(D, r);
                    }
                    if constexpr (BIG) {
                        float E[3][4];
                        fx_stack(E, fys, B, lane);
#pragma unroll
                        for (int b = 0; b < 2; b++) {
                            const long long v = fx_stack_value(E, b, g);
                            if (g >= 4 && 12 + g < N2 && 8 * tile + 2 * t + b < G::NC)
                                s_t[Zr[b] * PZ + (12 + g) * PX + Xr[b]] = v;
                        }
                    }
                }
                fx_landed();  // T2 (and A_z)
                if (j1 < ni) fx_copy(fsm + G::O_Y, s_py[j1] + G::X_Y, G::YW);
                // z pass over this warp's column tiles
                const uint32_t *fz0 = fsm + G::O_Z, *fzs = fz0 + G::TILEW;
                const int ez0 = s_exz[j0][g], ez1 = s_exz[j0][8 + g], ez2 = g >= 4 && BIG ? s_exz[j0][12 + g] : FX_NONE;
#pragma unroll 1
                for (int q = 0; q < G::TPW; q++) {
                    const int nt = warp + q * G::WARPS;
                    if (nt >= G::NT) continue;
                    const int c = 8 * nt + g;
                    int Yc, X;
                    fx_column<K>(min(c, G::NC - 1), Yc, X);
                    const long long *T = s_t + Yc * PX + X, *u = s_u + Yc * UX + X;
                    FxB B;
                    float D[10][4];
                    long long v[RA];
                    const bool in = c < G::NC;
                    fx_operand<K>(B, t, [&](int Z) -> long long { return !in || Z >= N2 ? 0 : T[Z * PZ]; });
                    fx_tile<BIG>(D, fz0, B, lane);
#pragma unroll
                    for (int r = 0; r < 4; r++) v[r] = fx_value(D, r);
                    if constexpr (BIG) {
                        float E[3][4];
                        fx_stack(E, fzs, B, lane);
#pragma unroll
                        for (int r = 0; r < 2; r++) v[4 + r] = fx_stack_value(E, r, g);
                    }
                    if (!root && nt < G::NTX) {  // scaling columns: the path without scaling-scaling where Z < K
                        const bool ins = c < K2;
                        fx_operand<K>(B, t, [&](int Z) -> long long { return !ins || Z >= N2 ? 0 : Z < K ? u[Z * UZ] : T[Z * PZ]; });
                        fx_tile<BIG>(D, fz0, B, lane);
#pragma unroll
                        for (int r = 0; r < 4; r++)
                            if (8 * nt + 2 * t + (r & 1) < K2 && g + 8 * (r >> 1) < K) v[r] = fx_value(D, r);
                    }
                    int ec[2];
#pragma unroll
                    for (int b = 0; b < 2; b++) {
                        int Yr, Xr;
                        fx_column<K>(min(8 * nt + 2 * t + b, G::NC - 1), Yr, Xr);
                        ec[b] = s_e1[par][Xr] + s_exy[j0][Yr];
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
                        s[r] = (up ? fx_round(acc[q][r], up) : acc[q][r]) + fx_round(v[r], eq - e[r]);
                        const int hi = (int)(s[r] >> 32);
                        over |= hi ^ (hi >> 31);
                    }
                    const int room = (over >> 29) ? 2 : 0;  // |sum| >= 2^61: make room for the next row's 2^62
                    ea[q] = eq + room;
#pragma unroll
                    for (int r = 0; r < RA; r++) acc[q][r] = fx_round(s[r], room);
                }
                nrows++;
                par ^= 1;
                j0 = j1;
            }
        }
        // a chunk's partial block is this task's alone; a whole node's block takes other tiers' sums too
        const bool set = L.set || (L.red_of && L.red_of[w] >= 0);
        double *out = L.out[w];
        const size_t cs = L.cstride ? L.cstride : (size_t)K3;
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
                double *o = out + (hq + 4 * hz) * cs + (Zq - hz * K) * K2 + (c - hq * K2);
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
void launch_to_fx(const FxSets &S, cudaStream_t s) {
    const int grid = (int)std::min<long long>(S.first[S.n], 65535);
    to_fx_kernel<K><<<grid, FxGeo<K>::THREADS, 0, s>>>(S);
    MWG_CUDA(cudaGetLastError());
}

template <int K>
void launch_op_to_fx(const FxOpJobs &jobs, int njobs, int most, cudaStream_t s) {
    const size_t smem = 4 * (size_t)FxGeo<K>::OP_WORDS;
    kernel_smem((const void *)op_to_fx_kernel<K>, (int)smem);
    op_to_fx_kernel<K><<<dim3(most, njobs), 32 * K, smem, s>>>(jobs);
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

size_t fx_op_words(int K) {
    switch (K) {
        case 4: return FxGeo<4>::OP_WORDS;
        case 5: return FxGeo<5>::OP_WORDS;
        case 6: return FxGeo<6>::OP_WORDS;
        case 7: return FxGeo<7>::OP_WORDS;
        case 8: return FxGeo<8>::OP_WORDS;
        case 9: return FxGeo<9>::OP_WORDS;
        case 10: return FxGeo<10>::OP_WORDS;
        default: throw Error(MW_ERR_ARG, "no fixed-point apply kernel for this order");
    }
}

size_t fx_op_z(int K) { return K > 8 ? FxGeo<10>::Z_OFF : FxGeo<8>::Z_OFF; }

void k_op_to_fx(const FxOpJob *jobs, size_t n, int K, cudaStream_t s) {
    for (size_t at = 0; at < n; at += FxOpJobs::MAX) {
        FxOpJobs J{};
        int m = 0, most = 0;
        for (; m < FxOpJobs::MAX && at + m < n; m++) {
            J.job[m] = jobs[at + m];
            most = std::max(most, J.job[m].n);
        }
        if (most == 0) continue;
        switch (K) {
            case 4: launch_op_to_fx<4>(J, m, most, s); break;
            case 5: launch_op_to_fx<5>(J, m, most, s); break;
            case 6: launch_op_to_fx<6>(J, m, most, s); break;
            case 7: launch_op_to_fx<7>(J, m, most, s); break;
            case 8: launch_op_to_fx<8>(J, m, most, s); break;
            case 9: launch_op_to_fx<9>(J, m, most, s); break;
            case 10: launch_op_to_fx<10>(J, m, most, s); break;
            default: throw Error(MW_ERR_ARG, "no fixed-point apply kernel for this order");
        }
    }
}

static void to_fx(const FxSets &S, int K, cudaStream_t s) {
    if (S.first[S.n] == 0) return;
    switch (K) {
        case 4: launch_to_fx<4>(S, s); break;
        case 5: launch_to_fx<5>(S, s); break;
        case 6: launch_to_fx<6>(S, s); break;
        case 7: launch_to_fx<7>(S, s); break;
        case 8: launch_to_fx<8>(S, s); break;
        case 9: launch_to_fx<9>(S, s); break;
        case 10: launch_to_fx<10>(S, s); break;
        default: throw Error(MW_ERR_ARG, "no fixed-point apply kernel for this order");
    }
}

void k_to_fx(const FxBlocks *sets, size_t n, int K, cudaStream_t s) {
    for (size_t at = 0; at < n; at += FxSets::MAX) {
        FxSets S{};
        for (; S.n < FxSets::MAX && at + S.n < n; S.n++) {
            const FxBlocks &b = sets[at + S.n];
            S.in[S.n] = b.in;
            S.out[S.n] = b.out;
            S.first[S.n + 1] = S.first[S.n] + (long long)b.n;
        }
        to_fx(S, K, s);
    }
}

void k_to_fx_list(const double *const *list, uint32_t *out, size_t n, int K, cudaStream_t s) {
    FxSets S{};
    S.n = 1;
    S.out[0] = out;
    S.first[1] = (long long)n;
    S.list = list;
    to_fx(S, K, s);
}

void k_pairs_to_fx(const PairTask *pairs, bool up, uint32_t *out, size_t n, int K, cudaStream_t s) {
    FxSets S{};
    S.n = 1;
    S.out[0] = out;
    S.first[1] = (long long)n;
    S.pairs = pairs;
    S.up = up ? 1 : 0;
    to_fx(S, K, s);
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

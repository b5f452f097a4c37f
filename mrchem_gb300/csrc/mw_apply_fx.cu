// mw_apply_fx.cu -- FP64-accuracy NS-form apply in 62-bit fixed point on the tensor cores.
//
// GB300's FP64 pipe runs 1.6 multiply-adds per SM and cycle, which bounds apply_kernel.  Here every
// operand of the three passes is a 62-bit fixed-point number with a power-of-two scale per row of an
// operator block and per column of the data, cut into seven signed 9-bit digits held as FP16
// integers: the error-free splitting of matrix products into low-precision ones that Ozaki et al. (Numer.
// Algorithms 59, 2012) describe.  A pass is a sum of 28 FP16 products (digit pairs i + j <= 6) on
// mma.sync.m16n8k16 with FP32 accumulation, and every sum is exact: see "ranges" below.
//
// Accuracy.  A column is brought to its own largest number before it is cut, in every pass: the dropped pairs
// (i + j >= 7) and the rounding of a result to 62 bits are below 2^-58 of (row 1-norm) x (column maximum).  Between
// the passes a number is held as 54 significant bits with its own exponent (fx_pack), so that no element loses bits
// to a larger one elsewhere in the block.  A node's sum has an exponent per row Z' and pair of columns.  What is
// left of the fixed scale is the column itself: a wavelet row of a narrow Gaussian takes little from the scaling half
// of a column and much from the small wavelet half.  The wavelet half of the data therefore counts 2^FX_UP times in a
// column's scale, and the operators' wavelet columns 2^-FX_UP: with 4 the small components of such items gain four
// bits and the scaling rows, nine bits better than FP64, lose none that FP64 has; with 7 and 9 they do.  In the
// results every component, the pure wavelet ones of far nodes too, is as close to the exact sums as apply_kernel's
// (at most 1.7 times its error, mostly less: tests/test_gpu_components.py).  With one exponent per X' for a whole
// block's intermediate and one per column tile for the node's sum, components that vanish beside the scaling part of
// a far node were off by 1e-6 of themselves.
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
// T is in shared memory, a 64-bit word per number (64 KB at 2K = 20), its row pitches 2 modulo 4 so that the rows 2t
// apart of one operand fall into distinct banks.  Digits are made where they serve many times: an input block's
// once per call, an operator block's once per level (op_to_fx_kernel; the z pass's with its term's
// coefficient), both laid out as mma.sync operands, the operators' copied to shared memory by cp.async one
// pass ahead.  Rows of items as in apply_kernel: a row's x passes add up, its y and z passes run once.
// Below the root scale the scaling-scaling path is left out exactly: u (wavelet-in-x part) comes from extra
// operator rows in the x pass's second row tile, and the (Y' < K, X' < K) columns of the z pass take a
// second operand whose Z < K part avoids that path.
//
// Measured over 16 Helmholtz applies at once (all of their levels, the nearly empty ones included), ns per item at
// 2K = 8, 10, .. 20: apply_kernel's FP64 pipe 30.9, 70.7, 116, 215, 308, 539, 797; this kernel 17.7, 35.8, 44.4, 65.3,
// 53.0, 150, 170.  Of that the numbers' own exponents between the passes take 0 to 7% (17.7, 35.5, 42.6, 67.3, 50.6,
// 140, 160 with common ones, which lost the small components).  Forms before, on a full chip at 2K = 20: T in
// registers and the operators' digits made per item 172, a row tile of their own for rows 16.. 147, then 134.
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
// Warps of a CTA: a divisor of the column tiles' number (50, 41, 32, 25, 18, 13, 8) with little left over, at
// most 16 (128 registers).  ns per item as above, this choice first:
//   K = 4: 8 warps, 2 CTAs per SM 17.7; 4, 4 CTAs 16.3; 8, 3 CTAs 16.3; 16, 1 CTA 24.8
//   K = 5: 7, 2 CTAs 35.8; 5, 3 CTAs 32.9; 7, 3 CTAs 37.1; 13, 1 CTA 46.4
//   K = 6: 9, 2 CTAs 44.4; 5, 3 CTAs 40.0; 9, 1 CTA 57.8
//   K = 7: 13, 1 CTA 65.3; 7, 2 CTAs 54.4; 9, 2 CTAs 55.2; 9, 1 CTA 71.8
//   K = 8: 8, 2 CTAs 53.0; 16, 1 CTA 61.9
// Fewer warps and more CTAs fill a loaded chip better, but a task then takes longer, which is what levels of few
// tasks wait for (K = 6 with 5 warps: 84 us a task against 70).  At 2K = 18, 20 shared memory holds one CTA; 17 warps
// at 2K = 20 (no nearly empty last round) spill: 146 ns against 134 in an earlier form.
constexpr int fx_warps(int K) { return K == 10 ? 16 : K == 9 ? 14 : K == 8 ? 8 : K == 7 ? 13 : K == 6 ? 9 : K == 5 ? 7 : 8; }

template <int K>
struct FxGeo {
    static constexpr int N2 = 2 * K, NC = N2 * N2, K2 = K * K, K3 = K2 * K;
    static constexpr bool BIG = N2 > 16;              // contraction remainder and a second row tile
    static constexpr int WARPS = fx_warps(K), THREADS = 32 * WARPS;
    static constexpr int MINB = K == 8 || K <= 6 ? 2 : 1;  // CTAs per SM that the registers are cut for
    // column tiles of the x pass: Y = 0..7, 8..15 of every plane Z; K > 8: Y >= 16 of two planes together
    static constexpr int CT = N2 > 8 ? 2 : 1, GRP = BIG ? K : N2, TL = BIG ? 5 : CT, NTIN = GRP * TL;
    // columns of the y and z passes: a component's K^2 and for odd K an empty one, so that the two columns of
    // a thread's results are of one component; their tiles, and those of them that take the second operand
    static constexpr int KE = K2 + (K2 & 1), NCE = 4 * KE, NT = (NCE + 7) / 8, NTX = (KE + 7) / 8;
    static constexpr int TPW = (NT + WARPS - 1) / WARPS;
    // T[Z][Y][X'] and u[Z][Y][X'] (Z, Y, X' < K), numbers as fx_pack has them
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
    // the columns' exponents (16 bits) and the largest of them
    static constexpr int WB = BIG ? 18 : 14, IN_EXP = NTIN * WB * 32, IN_MAX = IN_EXP + 4 * NTIN, IN_WORDS = IN_MAX + 4;
    // operator digits of a block: the x pass's (the y pass's from X_Y on) and the rows' exponents, the largest of
    // them in place EMAX; then those of the block times its term's coefficient (the z pass's)
    static constexpr int X_Y = TILEW, X_EXP = XW, Z_OFF = X_EXP + 16, Z_EXP = YW, OP_WORDS = Z_OFF + Z_EXP + 16;
    static_assert(Z_OFF == (BIG ? 2 * (7 + 10) + 14 : 2 * 7) * 128 + 16, "the same for all K of a kind");
    static_assert(O_U % 4 == 0 && O_X % 4 == 0 && TILEW % 4 == 0 && IN_WORDS % 4 == 0, "16-byte aligned copies");
};

constexpr float FX_MAGIC = 12582912.0f;  // 1.5 * 2^23
constexpr int FX_MAGIC_BITS = 0x4B400000;
constexpr int FX_SEG = 32;           // items whose pointers and exponents a CTA holds at a time
constexpr int FX_NONE = -20000;      // exponent of a zero row, column or block
constexpr int FX_EMAX = 31;          // place of a block's largest row exponent
constexpr int FX_UP = 4;             // data of the wavelet half count 2^FX_UP times, operators' wavelet columns 2^-FX_UP

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
    uint32_t ec;  // x pass: the exponents of the columns 2t and 2t + 1 of the results
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

// A number of the T arrays: 54 significant bits and in the low byte its binary places below the array's base B (a
// power of two that no number's unit exceeds).  v 2^(B - d - 62), |v| <= 2^62, d >= 0, to such a word; of what lies
// more than 255 places below the base, nothing is left that counts beside it.  The shift goes up to 30 places: a
// smaller v has no more than 32 bits that mean anything, and they all stay.
constexpr int FX_ZERO = 255;
__device__ __forceinline__ long long fx_pack(long long v, int d) {
    const int hi = (int)(v >> 32);
    const int n = max(__clz(hi ^ (hi >> 31)) - 2, 0), f = v ? min(d + n, 255) : FX_ZERO;
    return (((v << n) + 128) & ~255ll) | f;
}

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
        const double a = rows[it] * cf * (k >= K ? 1.0 / (1 << FX_UP) : 1.0);
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
        if (warp == 0) {
            short *exps = reinterpret_cast<short *>(fsm + G::X_EXP);
            const int e = __reduce_max_sync(0xffffffffu, lane < G::N2 ? (int)exps[lane] : FX_NONE);
            if (lane == 0) exps[FX_EMAX] = (short)e;
        }
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
// per column, for the blocks of several trees at once.  One CTA per block, a warp per tile.
template <int K>
__global__ void __launch_bounds__(FxGeo<K>::THREADS) to_fx_kernel(__grid_constant__ const FxSets S) {
    using G = FxGeo<K>;
    constexpr int N2 = G::N2, K2 = G::K2, K3 = G::K3;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const size_t cs = (size_t)(S.pairs && S.up ? 8 : 1) * K3;  // distance of a block's components
    const long long nb = S.first[S.n];
    __shared__ int s_most;
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
        if (threadIdx.x == 0) s_most = FX_NONE;
        __syncthreads();
        int most = FX_NONE;
        for (int tile = warp; tile < G::NTIN; tile += G::WARPS) {
            int Y, Z;
            fx_in_column<K>(tile / G::TL, tile % G::TL, g, Y, Z);
            // this lane's X of the column, every X in one lane (those of the remainder in two)
            constexpr int NX = G::BIG ? 6 : (N2 > 8 ? 4 : 2);
            double x[NX];
            auto col = [&](int j) { return j < 4 ? 2 * t + (j & 1) + 8 * (j >> 1) : 16 + 2 * (t & 1) + (j & 1); };
            int ef = 0;
#pragma unroll
            for (int j = 0; j < NX; j++) {
                x[j] = at(col(j), Y, Z);
                const int e = (__double2hiint(x[j]) >> 20) & 0x7ff;
                ef = max(ef, e == 0 ? 0 : e + (col(j) >= K ? FX_UP : 0));
            }
            ef = max(ef, __shfl_xor_sync(0xffffffffu, ef, 1));
            ef = max(ef, __shfl_xor_sync(0xffffffffu, ef, 2));
            const int ec = ef == 0 ? FX_NONE : ef - 1022;
            most = max(most, ec);
            if (t == 0) reinterpret_cast<short *>(o + G::IN_EXP)[8 * tile + g] = (short)ec;
            auto fixed = [&](int j) { return fx_from_double(x[j], ef - (col(j) >= K ? FX_UP : 0)); };
            uint32_t w[G::WB];
            uint32_t q[7];
            fx_digits(fixed(0), fixed(1), q);
#pragma unroll
            for (int s = 0; s < 7; s++) {
                w[2 * s] = q[s];
                w[2 * s + 1] = 0u;
            }
            if constexpr (N2 > 8) {
                fx_digits(fixed(2), fixed(3), q);
#pragma unroll
                for (int s = 0; s < 7; s++) w[2 * s + 1] = q[s];
            }
            if constexpr (G::BIG) {
                fx_digits(fixed(4), fixed(5), q);
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
        most = __reduce_max_sync(0xffffffffu, most);
        if (lane == 0) atomicMax(&s_most, most);
        __syncthreads();
        if (threadIdx.x == 0) o[G::IN_MAX] = (uint32_t)s_most;
        __syncthreads();
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
    asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(B.ec) : "l"(blk + G::IN_EXP + 4 * tile + (lane & 3)));
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

// One lane's operand of a y- or z-pass tile: word(k) is the column's k-th number (fx_pack), FX_ZERO for k >= 2K.
// The column's numbers are brought to the largest one's places: returned, for the digits' scale 2^(B - places).
template <int K, typename F>
__device__ __forceinline__ int fx_operand(FxB &B, int t, F word) {
    using G = FxGeo<K>;
    constexpr int NE = G::BIG ? 6 : (G::N2 > 8 ? 4 : 2);
    long long m[NE];
    int f[NE], places = 1000;
#pragma unroll
    for (int j = 0; j < NE; j++) {
        const int k = j < 4 ? 2 * t + (j & 1) + 8 * (j >> 1) : 16 + 2 * (t & 1) + (j & 1);
        const long long w = word(k);
        f[j] = (int)(w & 255) - (k >= K ? FX_UP : 0);
        m[j] = w & ~255ll;
        places = min(places, f[j]);
    }
    places = min(places, __shfl_xor_sync(0xffffffffu, places, 1));
    places = min(places, __shfl_xor_sync(0xffffffffu, places, 2));
    uint32_t q[7];
    fx_digits(fx_round(m[0], f[0] - places), fx_round(m[1], f[1] - places), q);
#pragma unroll
    for (int s = 0; s < 7; s++) B.m[s][0] = q[s];
    if constexpr (NE > 2) {
        fx_digits(fx_round(m[2], f[2] - places), fx_round(m[3], f[3] - places), q);
#pragma unroll
        for (int s = 0; s < 7; s++) B.m[s][1] = q[s];
    } else {
#pragma unroll
        for (int s = 0; s < 7; s++) B.m[s][1] = 0u;
    }
    if constexpr (NE > 4) {
        fx_digits(fx_round(m[4], f[4] - places), fx_round(m[5], f[5] - places), q);
        B.fold(q, t >= 2);
    }
    return places;
}

// column c of the y pass (a = Z) or z pass (a = Y'): the scaling columns (a < K, X' < K) first; false for an empty one
template <int K>
__device__ __forceinline__ bool fx_column(int c, int &a, int &x) {
    using G = FxGeo<K>;
    const int q = min(c / G::KE, 3), r = min(c - q * G::KE, G::K2 - 1), i = r / K;
    a = (q >> 1) * K + i;
    x = (q & 1) * K + r - i * K;
    return c < G::NCE && c - q * G::KE < G::K2;
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
    __shared__ int s_node, s_redf, s_most[FX_SEG];  // s_most: the input blocks' largest exponents
    __shared__ const uint32_t *s_pi[FX_SEG], *s_px[FX_SEG], *s_py[FX_SEG], *s_pz[FX_SEG];
    __shared__ short s_exx[FX_SEG][32], s_exy[FX_SEG][32], s_exz[FX_SEG][32];  // row exponents
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const bool root = L.root != 0;
    // the rows of this lane's results: g, 8 + g and, in the second row tile, 12 + g (g >= 4) or u's 8 + g
    const int x2 = g >= 4 ? 12 + g : 8 + g;

    while (true) {
        __syncthreads();
        if (tid == 0) s_node = atomicAdd(L.counter, 1);
        __syncthreads();
        const int w = s_node;
        if (w >= L.nnodes) break;
        const long long b0 = L.begin[w], b1 = L.end[w];
        // node accumulator: per column tile of this warp (columns 8 nt + 2t, + 1) rows Z' = g, 8 + g, 12 + g
        // (g >= 4), each row of a thread in units of 2^(ea - 62).  Indexed in a rolled loop, so it lives in
        // local memory between the z passes.
        long long acc[G::TPW][RA];
        int ea[G::TPW][RA / 2];
#pragma unroll 1
        for (int q = 0; q < G::TPW; q++)
            for (int r = 0; r < RA; r++) {
                ea[q][r / 2] = -1000000;
                acc[q][r] = 0;
            }
        int nrows = 0;
        for (long long sb = b0; sb < b1; sb += FX_SEG) {
            const int ni = (int)min((long long)FX_SEG, b1 - sb);
            if (sb != b0) __syncthreads();
            for (int i = tid; i < ni; i += G::THREADS) {
                s_pi[i] = reinterpret_cast<const uint32_t *>(L.in[sb + i]);
                s_px[i] = reinterpret_cast<const uint32_t *>(L.ax[sb + i]);
                s_py[i] = reinterpret_cast<const uint32_t *>(L.ay[sb + i]);
                s_pz[i] = reinterpret_cast<const uint32_t *>(L.az[sb + i]);
                s_most[i] = (int)s_pi[i][G::IN_MAX];
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
            const uint32_t *lastz = nullptr;
            for (int j0 = 0; j0 < ni;) {
                int j1 = j0 + 1;  // the row: items of one term, ly and lz
                while (j1 < ni && s_py[j1] == s_py[j0] && s_pz[j1] == s_pz[j0]) j1++;
                int base = 0;  // of T1 and u: no item's units nor their sums' exceed it
                for (int j = j0; j < j1; j++) {
                    const bool first = j == j0;
                    const uint32_t *in = s_pi[j];
                    FxB B, Bn;
                    if (warp < G::NTIN) fx_load<K>(Bn, in, warp, lane);
                    fx_landed();  // A_x (and A_y); the z pass has read T
                    if (first) {
                        if (s_pz[j0] != lastz) {  // rows of one term and lz share A_z
                            lastz = s_pz[j0];
                            fx_copy(fsm + G::O_Z, lastz, G::YW);
                        }
                        base = s_most[j0] + s_exx[j0][FX_EMAX];
                        for (int i = j0 + 1; i < j1; i++) base = max(base, s_most[i] + s_exx[i][FX_EMAX]);
                        if (j1 - j0 > 1) base += 34 - __clz(j1 - j0 - 1);  // the sums' bits, and one for each addition's room
                    }
                    // places of the rows' units below the base, less the column's exponent
                    const int dg = base - s_exx[j][g], dh = base - s_exx[j][8 + g], dq = base - s_exx[j][x2];
                    const uint32_t *fx1 = fsm + G::O_X + (j & 1) * G::XW, *fx0 = fx1 + G::X_Y, *fxs = fx0 + G::TILEW;
                    if (j + 1 < ni) fx_copy(fsm + G::O_X + ((j + 1) & 1) * G::XW, s_px[j + 1], G::XW);
                    // the row's first item, which stores, has code of its own: with the additions in the same loop an
                    // item took 2 to 4% longer (170 and 174 ns at 2K = 20)
                    auto x_pass = [&](auto one) {
                        constexpr bool ONE = decltype(one)::value;
#pragma unroll 1
                        for (int tile = warp; tile < G::NTIN; tile += G::WARPS) {
                            B = Bn;  // the next tile's operand comes from L2 behind this one's products
                            if (tile + G::WARPS < G::NTIN) fx_load<K>(Bn, in, tile + G::WARPS, lane);
                            const int gr = tile / G::TL, ti = tile - gr * G::TL;
                            const int ec[2] = {(int)(short)(B.ec & 0xffffu), (int)B.ec >> 16};
                            // the row's sum so far and this item's result, in the coarser unit with one bit of room
                            auto add = [&](long long *s, long long v, int d) {
                                if constexpr (!ONE) {
                                    const long long o = *s;
                                    const int f = (int)(o & 255), to = min(d, f) - 1;
                                    v = fx_round(v, d - to) + fx_round(o & ~255ll, f - to);
                                    d = to;
                                }
                                *s = fx_pack(v, d);
                            };
                            int Y, Z;  // of column 2t; column 2t + 1 is Y + 1
                            fx_in_column<K>(gr, ti, 2 * t, Y, Z);
                            long long *T = s_t + Z * PZ + Y * PX, *u = s_u + Z * UZ + Y * UX;
                            float D[10][4];
                            fx_tile<BIG>(D, fx0, B, lane);
#pragma unroll
                            for (int r = 0; r < 4; r++)
                                if (g + 8 * (r >> 1) < N2 && Y + (r & 1) < N2)
                                    add(T + (r & 1) * PX + g + 8 * (r >> 1), fx_value(D, r), (r < 2 ? dg : dh) - ec[r & 1]);
                            const bool has_u = !root && Z < K && Y < K;
                            if (BIG && (root || ti == 4 || 2 * gr + ti / 2 >= K)) {  // no column with u (the warp's tile as a whole)
                                float E[3][4];
                                fx_stack(E, fxs, B, lane);
#pragma unroll
                                for (int r = 0; r < 2; r++) {
                                    const long long v = fx_stack_value(E, r, g);
                                    if (g >= 4 && 12 + g < N2 && Y + r < N2) add(T + r * PX + 12 + g, v, dq - ec[r]);
                                }
                            } else if constexpr (BIG) {
                                fx_tile<BIG>(D, fx1, B, lane);
#pragma unroll
                                for (int r = 0; r < 2; r++) {
                                    if (g >= 4 && 12 + g < N2 && Y + r < N2) add(T + r * PX + 12 + g, fx_value(D, r), dq - ec[r]);
                                    if (g < 2 && 8 + g < K && has_u && Y + r < K) add(u + r * UX + 8 + g, fx_value(D, r), dq - ec[r]);
                                    if (has_u && Y + r < K) add(u + r * UX + g, fx_value(D, 2 + r), dg - ec[r]);
                                }
                            } else if (!root && ti == 0 && gr < K) {
                                fx_tile<BIG>(D, fx1, B, lane);
#pragma unroll
                                for (int r = 0; r < 2; r++)
                                    if (g < K && Y + r < K) add(u + r * UX + g, fx_value(D, r), dg - ec[r]);
                            }
                        }
                    };
                    if (first)
                        x_pass(std::true_type());
                    else
                        x_pass(std::false_type());
                }
                fx_landed();
                // y pass in place: a warp reads its 8 columns (Z, X') whole before it writes them
                const int base2 = base + FX_UP + s_exy[j0][FX_EMAX];  // of T2
                const int yg = base2 - base - s_exy[j0][g], yh = base2 - base - s_exy[j0][8 + g],
                          yq = base2 - base - s_exy[j0][x2];
                const uint32_t *fy0 = fsm + G::O_Y, *fys = fy0 + G::TILEW;
#pragma unroll 1
                for (int tile = warp; tile < G::NT; tile += G::WARPS) {
                    int Z, X;
                    const bool in = fx_column<K>(8 * tile + g, Z, X);
                    const long long *T = s_t + Z * PZ + X, *u = s_u + Z * UZ + X;
                    int Zr[2], Xr[2], at[2];  // of the results' columns 2t, 2t + 1, and the places of their scales
                    bool inr[2];
#pragma unroll
                    for (int b = 0; b < 2; b++) inr[b] = fx_column<K>(8 * tile + 2 * t + b, Zr[b], Xr[b]);
                    FxB B;
                    float D[10][4];
                    if (!root && tile < G::NTX) {  // scaling columns: u where Y < K
                        const bool s = in && Z < K && X < K;
                        const int p = fx_operand<K>(B, t, [&](int Y) -> long long {
                            return !s || Y >= N2 ? FX_ZERO : Y < K ? u[Y * UX] : T[Y * PX];
                        });
#pragma unroll
                        for (int b = 0; b < 2; b++) at[b] = __shfl_sync(0xffffffffu, p, 4 * (2 * t + b));
                        fx_tile<BIG>(D, fy0, B, lane);
                        __syncwarp();
#pragma unroll
                        for (int r = 0; r < 4; r++) {
                            const int Yq = g + 8 * (r >> 1), b = r & 1;
                            if (Yq < K && inr[b] && Zr[b] < K && Xr[b] < K)
                                s_u[Zr[b] * UZ + Yq * UX + Xr[b]] = fx_pack(fx_value(D, r), (r < 2 ? yg : yh) + at[b]);
                        }
                    }
                    const int p = fx_operand<K>(B, t, [&](int Y) -> long long { return !in || Y >= N2 ? FX_ZERO : T[Y * PX]; });
#pragma unroll
                    for (int b = 0; b < 2; b++) at[b] = __shfl_sync(0xffffffffu, p, 4 * (2 * t + b));
                    fx_tile<BIG>(D, fy0, B, lane);
                    __syncwarp();
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const int Yq = g + 8 * (r >> 1), b = r & 1;
                        if (Yq < N2 && inr[b])
                            s_t[Zr[b] * PZ + Yq * PX + Xr[b]] = fx_pack(fx_value(D, r), (r < 2 ? yg : yh) + at[b]);
                    }
                    if constexpr (BIG) {
                        float E[3][4];
                        fx_stack(E, fys, B, lane);
#pragma unroll
                        for (int b = 0; b < 2; b++) {
                            const long long v = fx_stack_value(E, b, g);
                            if (g >= 4 && 12 + g < N2 && inr[b]) s_t[Zr[b] * PZ + (12 + g) * PX + Xr[b]] = fx_pack(v, yq + at[b]);
                        }
                    }
                }
                fx_landed();  // T2 (and A_z)
                if (j1 < ni) fx_copy(fsm + G::O_Y, s_py[j1] + G::X_Y, G::YW);
                // z pass over this warp's column tiles
                const uint32_t *fz0 = fsm + G::O_Z, *fzs = fz0 + G::TILEW;
                const int ez[3] = {base2 + s_exz[j0][g], base2 + s_exz[j0][8 + g],
                                   g >= 4 && BIG ? base2 + s_exz[j0][12 + g] : 2 * FX_NONE};
#pragma unroll 1
                for (int q = 0; q < G::TPW; q++) {
                    const int nt = warp + q * G::WARPS;
                    if (nt >= G::NT) continue;
                    int Yc, X;
                    const bool in = fx_column<K>(8 * nt + g, Yc, X);
                    const long long *T = s_t + Yc * PX + X, *u = s_u + Yc * UX + X;
                    FxB B;
                    float D[10][4];
                    long long v[RA];
                    int e[RA];
                    int p = fx_operand<K>(B, t, [&](int Z) -> long long { return !in || Z >= N2 ? FX_ZERO : T[Z * PZ]; });
                    fx_tile<BIG>(D, fz0, B, lane);
#pragma unroll
                    for (int r = 0; r < 4; r++) v[r] = fx_value(D, r);
                    if constexpr (BIG) {
                        float E[3][4];
                        fx_stack(E, fzs, B, lane);
#pragma unroll
                        for (int r = 0; r < 2; r++) v[4 + r] = fx_stack_value(E, r, g);
                    }
#pragma unroll
                    for (int b = 0; b < 2; b++) {
                        const int at = __shfl_sync(0xffffffffu, p, 4 * (2 * t + b));
#pragma unroll
                        for (int r = b; r < RA; r += 2) e[r] = ez[r >> 1] - at;
                    }
                    if (!root && nt < G::NTX) {  // scaling columns: the path without scaling-scaling where Z < K
                        const bool s = in && Yc < K && X < K;
                        p = fx_operand<K>(B, t, [&](int Z) -> long long { return !s || Z >= N2 ? FX_ZERO : Z < K ? u[Z * UZ] : T[Z * PZ]; });
                        fx_tile<BIG>(D, fz0, B, lane);
#pragma unroll
                        for (int b = 0; b < 2; b++) {
                            const int at = __shfl_sync(0xffffffffu, p, 4 * (2 * t + b));
                            int Yr, Xr;
                            if (!fx_column<K>(8 * nt + 2 * t + b, Yr, Xr) || Yr >= K || Xr >= K) continue;
#pragma unroll
                            for (int r = b; r < 4; r += 2)
                                if (g + 8 * (r >> 1) < K) {
                                    v[r] = fx_value(D, r);
                                    e[r] = ez[r >> 1] - at;
                                }
                        }
                    }
#pragma unroll
                    for (int r = 0; r < RA; r += 2) {
                        const int eq = max(ea[q][r / 2], max(e[r], e[r + 1])), up = eq - ea[q][r / 2];
                        long long s0 = acc[q][r], s1 = acc[q][r + 1];
                        if (up) {
                            s0 = fx_round(s0, up);
                            s1 = fx_round(s1, up);
                        }
                        s0 += fx_round(v[r], eq - e[r]);
                        s1 += fx_round(v[r + 1], eq - e[r + 1]);
                        const int h0 = (int)(s0 >> 32), h1 = (int)(s1 >> 32);
                        // |sum| >= 2^61: make room for the next row's 2^62
                        const int room = (((h0 ^ (h0 >> 31)) | (h1 ^ (h1 >> 31))) >> 29) ? 2 : 0;
                        ea[q][r / 2] = eq + room;
                        acc[q][r] = fx_round(s0, room);
                        acc[q][r + 1] = fx_round(s1, room);
                    }
                }
                nrows++;
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
                const int hq = c / G::KE, hz = Zq >= K;
                if (c >= G::NCE || c - hq * G::KE >= K2 || Zq >= N2) continue;
                const double v = fx_to_double(acc[q][r], ea[q][r / 2] - 62);
                double *o = out + (hq + 4 * hz) * cs + (Zq - hz * K) * K2 + (c - hq * G::KE);
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

// mw_opbuild.cu -- the non-standard-form blocks of a separated-Gaussian operator, built on the GPU.
//
// For term t (exponent a) at scale n (s = n + 1) the 1-D NS block of translation l is
//   NS_n(l) = W [[tau(2l), tau(2l-1)], [tau(2l+1), tau(2l)]] W^T,
//   tau(m)_ij = 2^-s int int phi_i(u) phi_j(v) exp(-a 4^-s (u - v + m)^2) du dv,
// evaluated through the Legendre expansion of the scaling functions' cross-correlation (degree
// 2K-1, coefficients prepared on the host) against Gaussian moments
//   G[p] = int_0^1 P_p(2z-1) exp(-beta (z + m)^2) dz
// by composite 16-point Gauss-Legendre quadrature, as the host construction does (mw_basis.cpp).
//
// Phase 1 walks l = 0, 1, ... of every (term, scale), writes the four sub-block norms of each NS(l) and
// stops where the host construction stops: the band follows from them.  It keeps the blocks of the first
// translations.  Phase 2 (one CTA per (term, scale, l) inside the band) zeroes the sub-blocks the host
// marked, and writes NS(l) and NS(-l) = NS(l)^T at their final places.  All arithmetic is FP64 in a fixed
// order, so the blocks are reproducible.
#include <algorithm>

#include "mw_host.h"

namespace mwg {

namespace {

constexpr int OB_THREADS = 128;
constexpr int OB_QPTS = 16;
constexpr int OB_UNIT = 8 * OB_QPTS;  // points of the 8 panels of a kernel wide against [0, 1]

// Shared memory of one CTA, K known at compile time (K = 10: 45 KB, five CTAs per SM).
template <int K>
struct ObShared {
    static constexpr int N2 = 2 * K;
    double P[OB_UNIT][N2 + 1];  // P_p(2z-1) at the points of 8 panels on [0, 1]; an odd pitch
    double W[N2 * N2];
    double G[3][N2];            // moments of 2l-1, 2l, 2l+1
    double H[4][N2];            // two moments, each in halves
    double tm1[K * K], t0[K * K], tp1[K * K];
    double T1[N2 * N2], ns[N2 * N2];
    double nrm[4];
    double gx[OB_QPTS], gw[OB_QPTS];
};

// P_0..P_{2K-1} at t by the three-term recurrence
template <int N2>
__device__ __forceinline__ void ob_legendre(double t, double (&P)[N2]) {
    P[0] = 1.0;
    P[1] = t;
#pragma unroll
    for (int j = 1; j + 1 < N2; j++) P[j + 1] = ((2.0 * j + 1.0) / (j + 1.0)) * t * P[j] - (j / (j + 1.0)) * P[j - 1];
}

// One warp: half the points' share of G_m[p] = int_0^1 P_p(2z-1) exp(-beta (z + m)^2) dz, to S.H[slot].  The
// lanes share the points out; their partial sums are added by a fixed order of exchanges, after each of
// which a lane keeps half of the values, so that lane p ends with the sum for p.  A kernel wide enough for 8
// panels on all of [0, 1] takes its Legendre values from the table.
template <int K>
__device__ void ob_moments(double beta, double l, int half, int slot, ObShared<K> &S) {
    constexpr int N2 = 2 * K;
    const int lane = threadIdx.x & 31;
    double acc[N2];
#pragma unroll
    for (int p = 0; p < N2; p++) acc[p] = 0.0;
    const double c0 = -l, w = 1.0 / sqrt(beta);
    const double lo = fmax(0.0, c0 - 12.0 * w), hi = fmin(1.0, c0 + 12.0 * w);
    if (lo < hi) {
        const double pw = fmin(0.125, 0.5 * w);
        const int npc = (int)ceil((hi - lo) / pw);
        const double step = (hi - lo) / npc;
        const bool unit = npc == 8 && lo == 0.0 && hi == 1.0;
        for (int i = 32 * half + lane; i < npc * OB_QPTS; i += 64) {
            const int k = i / OB_QPTS, q = i - k * OB_QPTS;
            const double z = (lo + k * step) + step * S.gx[q], e = beta * (z + l) * (z + l);
            if (e > 745.0) continue;
            const double g = step * S.gw[q] * exp(-e);
            if (unit) {
#pragma unroll
                for (int p = 0; p < N2; p++) acc[p] += g * S.P[i][p];
            } else {
                double P[N2];
                ob_legendre<N2>(2.0 * z - 1.0, P);
#pragma unroll
                for (int p = 0; p < N2; p++) acc[p] += g * P[p];
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int j = 0; j < o; j++) {
            if (j >= N2) continue;
            const double high = j + o < N2 ? acc[(j + o) % N2] : 0.0;
            const double got = __shfl_xor_sync(0xffffffffu, up ? acc[j] : high, o);
            acc[j] = (up ? high : acc[j]) + got;
        }
    }
    if (lane < N2) S.H[slot][lane] = acc[0];
}

// All threads: S.G[1] = G_m and S.G[2] = G_{m+1}, S.G[0] = the last S.G[2].  Two warps per moment.
template <int K>
__device__ void ob_pair(double beta, int m, ObShared<K> &S) {
    const int q = threadIdx.x >> 5, p = threadIdx.x;
    ob_moments<K>(beta, (double)(m + (q >> 1)), q & 1, q, S);
    __syncthreads();
    if (p < 2 * K) {
        S.G[0][p] = S.G[2][p];
        S.G[1][p] = S.H[0][p] + S.H[1][p];
        S.G[2][p] = S.H[2][p] + S.H[3][p];
    }
    __syncthreads();
}

// out = tau(m) (K x K) from the moments of m and -m, each as it is or (odd) its mirror image: with z -> 1 - z,
// G_{-m}[p] = (-1)^p G_{m-1}[p]
template <int K>
__device__ __forceinline__ void ob_tau(double pref, const double *cc, const double *gp, bool odd_p, const double *gm,
                                       bool odd_m, double *out) {
    constexpr int N2 = 2 * K;
    for (int e = threadIdx.x; e < K * K; e += OB_THREADS) {
        const int i = e / K, j = e - i * K;
        const double *aij = cc + (size_t)(i * K + j) * N2, *aji = cc + (size_t)(j * K + i) * N2;
        double even = 0.0, up = 0.0, um = 0.0;  // even p, odd p of both
#pragma unroll
        for (int p = 0; p < N2; p += 2) {
            even += __ldg(aij + p) * gp[p] + __ldg(aji + p) * gm[p];
            up += __ldg(aij + p + 1) * gp[p + 1];
            um += __ldg(aji + p + 1) * gm[p + 1];
        }
        out[e] = pref * (even + ((odd_p ? -up : up) + (odd_m ? -um : um)));
    }
}

// S.ns = W [[t0, tm1], [tp1, t0]] W^T and its four sub-block norms, all threads call
template <int K>
__device__ void ob_ns(ObShared<K> &S) {
    constexpr int N2 = 2 * K;
    for (int e = threadIdx.x; e < N2 * N2; e += OB_THREADS) {
        const int r = e / N2, c = e - r * N2, j = c % K;
        const double *up = c < K ? S.t0 : S.tm1, *dn = c < K ? S.tp1 : S.t0;
        double v = 0.0;
#pragma unroll
        for (int k = 0; k < K; k++) v += S.W[r * N2 + k] * up[k * K + j];
#pragma unroll
        for (int k = 0; k < K; k++) v += S.W[r * N2 + K + k] * dn[k * K + j];
        S.T1[e] = v;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < N2 * N2; e += OB_THREADS) {
        const int r = e / N2, c = e - r * N2;
        double v = 0.0;
#pragma unroll
        for (int k = 0; k < N2; k++) v += S.T1[r * N2 + k] * S.W[c * N2 + k];
        S.ns[e] = v;
    }
    __syncthreads();
    {  // a warp per sub-block
        const int q = threadIdx.x >> 5, lane = threadIdx.x & 31, g = q >> 1, f = q & 1;
        double s = 0.0;
        for (int e = lane; e < K * K; e += 32) {
            const double v = S.ns[(g * K + e / K) * N2 + f * K + e % K];
            s += v * v;
        }
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) S.nrm[q] = sqrt(s);
    }
    __syncthreads();
}

template <int K>
__device__ void ob_setup(const double *W, const double *gx, const double *gw, ObShared<K> &S) {
    constexpr int N2 = 2 * K;
    if (threadIdx.x < OB_QPTS) {
        S.gx[threadIdx.x] = gx[threadIdx.x];
        S.gw[threadIdx.x] = gw[threadIdx.x];
    }
    for (int e = threadIdx.x; e < N2 * N2; e += OB_THREADS) S.W[e] = W[e];
    __syncthreads();
    for (int i = threadIdx.x; i < OB_UNIT; i += OB_THREADS) {
        double P[N2];
        ob_legendre<N2>(2.0 * (0.125 * (i / OB_QPTS) + 0.125 * S.gx[i % OB_QPTS]) - 1.0, P);
        for (int p = 0; p < N2; p++) S.P[i][p] = P[p];
    }
    __syncthreads();
}

// tau(2l-1), tau(2l), tau(2l+1) of block l; `next`: the last block was l - 1, whose tau(2l+1) and moment are
// this one's tau(2l-1) and G_{2l-1}.  Two moments per block: those of -2l and -(2l+1) are the mirror images of
// G_{2l-1} and G_{2l}.
template <int K>
__device__ void ob_taus(const OpBuildTask &T, int l, bool next, const double *cc, ObShared<K> &S) {
    if (l > 0) {
        if (next) {
            for (int e = threadIdx.x; e < K * K; e += OB_THREADS) S.tm1[e] = S.tp1[e];
        } else {
            ob_pair<K>(T.beta, 2 * l - 2, S);
            ob_tau<K>(T.pref, cc, S.G[2], false, S.G[1], true, S.tm1);
            __syncthreads();
        }
    }
    ob_pair<K>(T.beta, 2 * l, S);
    ob_tau<K>(T.pref, cc, S.G[1], false, l > 0 ? S.G[0] : S.G[1], l > 0, S.t0);
    ob_tau<K>(T.pref, cc, S.G[2], false, S.G[1], true, S.tp1);
    if (l == 0) ob_tau<K>(T.pref, cc, S.G[1], true, S.G[2], false, S.tm1);
    __syncthreads();
}

// Phase 1: per task the sub-block norms of NS(0..L) and L, where the walk stops; the blocks themselves for
// l < OP_KEEP, which most walks do not pass.  Persistent CTAs.  Bound: the FP64 pipe (per block 2 (2K)^3
// multiply-adds for W tau W^T, 8 K^3 for the two taus, and two moments of at most 128 points with an exponential
// and 2K multiply-adds each).  8 Helmholtz operators of order 9: 3.8 ms; 5.4 ms with the moments of negative
// translations computed too and every lane adding every partial sum.
template <int K>
__global__ void __launch_bounds__(OB_THREADS) op_band_kernel(const double *W, const double *cc, const double *gx,
                                                             const double *gw, const OpBuildTask *tasks, int ntask,
                                                             double *nrm, double *head, int *band, double *peak,
                                                             double *keep) {
    extern __shared__ __align__(16) unsigned char ob_smem[];
    ObShared<K> &S = *reinterpret_cast<ObShared<K> *>(ob_smem);
    ob_setup<K>(W, gx, gw, S);
    for (int t = blockIdx.x; t < ntask; t += gridDim.x) {
        const OpBuildTask T = tasks[t];
        double *tn = nrm + T.nrm_off;
        double pk = 0.0;
        int L = -1;
        for (int l = 0; l <= T.cap; l++) {
            ob_taus<K>(T, l, true, cc, S);
            ob_ns<K>(S);
            if (threadIdx.x < 4) {
                tn[4 * l + threadIdx.x] = S.nrm[threadIdx.x];
                if (l < OP_NRM_HEAD) head[((size_t)t * OP_NRM_HEAD + l) * 4 + threadIdx.x] = S.nrm[threadIdx.x];
            }
            if (l < OP_KEEP)
                for (int e = threadIdx.x; e < 4 * K * K; e += OB_THREADS)
                    keep[((size_t)t * OP_KEEP + l) * 4 * K * K + e] = S.ns[e];
            L = l;
            bool stop = false;
            if (!T.root) {
                const double mx = fmax(fmax(S.nrm[0], S.nrm[1]), fmax(S.nrm[2], S.nrm[3]));
                const double nsn = fmax(S.nrm[1], fmax(S.nrm[2], S.nrm[3]));
                if (l <= 1) pk = fmax(pk, mx);
                if (l >= 2 && nsn < NS_CLEAN * pk) {
                    L = l - 1;
                    stop = true;
                }
            }
            __syncthreads();
            if (stop) break;
        }
        if (threadIdx.x == 0) {
            band[t] = L;
            peak[t] = pk;
        }
    }
}

// Phase 2: block l of task `task` (one CTA per (task, l) pair), kept by phase 1 or, from OP_KEEP on, computed
// again; zero: 4 bits, sub-blocks to zero.
template <int K>
__global__ void __launch_bounds__(OB_THREADS) op_block_kernel(const double *W, const double *cc, const double *gx,
                                                              const double *gw, const OpBuildTask *tasks,
                                                              const OpBlockJob *jobs, int njob, const double *keep) {
    extern __shared__ __align__(16) unsigned char ob_smem[];
    ObShared<K> &S = *reinterpret_cast<ObShared<K> *>(ob_smem);
    constexpr int N2 = 2 * K, bsz = N2 * N2;
    bool set = false;
    for (int q = blockIdx.x; q < njob; q += gridDim.x) {
        const OpBlockJob J = jobs[q];
        const int l = J.l;
        __syncthreads();
        if (l < OP_KEEP) {
            const double *k = keep + ((size_t)J.task * OP_KEEP + l) * bsz;
            for (int e = threadIdx.x; e < bsz; e += OB_THREADS) S.ns[e] = k[e];
        } else {
            if (!set) ob_setup<K>(W, gx, gw, S);
            set = true;
            ob_taus<K>(tasks[J.task], l, false, cc, S);
            ob_ns<K>(S);
        }
        __syncthreads();
        double *pos = J.blocks + (size_t)(J.off + J.band + l) * bsz;
        double *neg = J.blocks + (size_t)(J.off + J.band - l) * bsz;
        for (int e = threadIdx.x; e < bsz; e += OB_THREADS) {
            const int r = e / N2, c = e - r * N2, g = r / K, f = c / K;
            pos[e] = (J.zero >> (2 * g + f)) & 1 ? 0.0 : S.ns[e];
            // NS(-l) = NS(l)^T, written in its own order
            if (l > 0) neg[e] = (J.zero >> (2 * f + g)) & 1 ? 0.0 : S.ns[c * N2 + r];
        }
    }
}

// FP32 copy of every block, and the tensor-core tier's B operand (mw_tc05_layout.h)
// round to TF32: nearest, ties away from zero (infinities and NaNs unchanged)
__device__ __forceinline__ float tf32_round(float v) {
    uint32_t u = __float_as_uint(v);
    if ((u & 0x7f800000u) != 0x7f800000u) u = (u + 0x1000u) & ~0x1fffu;
    return __uint_as_float(u);
}

__global__ void op_convert_kernel(const double *blocks, float *b32, float *btc, float *btc2, long nblocks, int K,
                                  int NB, int groups) {
    const int N2 = 2 * K, bsz = N2 * N2;
    const size_t total = (size_t)nblocks * bsz;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x)
        b32[i] = __double2float_rn(blocks[i]);
    if (!btc) return;
    // per block: the B operand rounded to TF32 (hi), then the remainder rounded to TF32 (lo)
    const size_t per = (size_t)groups * NB * 4, ttot = (size_t)nblocks * per;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < ttot; i += (size_t)gridDim.x * blockDim.x) {
        const size_t blk = i / per;
        const int rem = (int)(i - blk * per), g = rem / (NB * 4), n = (rem / 4) % NB, c = rem % 4, k = 4 * g + c;
        double d = 0.0;
        if (k < N2) {
            const size_t base = blk * bsz;
            if (n < N2)
                d = blocks[base + (size_t)n * N2 + k];
            else if (n < N2 + K && k >= K)
                d = blocks[base + (size_t)(n - N2) * N2 + k];
        }
        const float h = tf32_round(__double2float_rn(d));
        const float l = tf32_round(__double2float_rn(d - (double)h));
        btc[2 * blk * per + rem] = h;
        btc[2 * blk * per + per + rem] = l;
        if (btc2) {  // the split tier's layout: per k-group its NB hi rows, then its NB lo rows
            const size_t gb = 2 * blk * per + (size_t)g * 2 * NB * 4 + (size_t)(rem % (NB * 4));
            btc2[gb] = h;
            btc2[gb + NB * 4] = l;
        }
    }
}

}  // namespace

namespace {

template <int K>
void launch_band(const double *W, const double *cc, const double *gx, const double *gw, const OpBuildTask *tasks,
                 int ntask, double *nrm, double *head, int *band, double *peak, double *keep, int nsm, cudaStream_t s) {
    const int smem = (int)sizeof(ObShared<K>);
    kernel_smem((const void *)op_band_kernel<K>, smem);
    const int per = std::max(1, kernel_ctas_per_sm((const void *)op_band_kernel<K>, OB_THREADS, smem));
    op_band_kernel<K><<<std::min(ntask, per * std::max(nsm, 1)), OB_THREADS, smem, s>>>(W, cc, gx, gw, tasks, ntask, nrm,
                                                                                     head, band, peak, keep);
    MWG_CUDA(cudaGetLastError());
}

template <int K>
void launch_blocks(const double *W, const double *cc, const double *gx, const double *gw, const OpBuildTask *tasks,
                   const OpBlockJob *jobs, int njob, const double *keep, cudaStream_t s) {
    const int smem = (int)sizeof(ObShared<K>);
    kernel_smem((const void *)op_block_kernel<K>, smem);
    op_block_kernel<K><<<std::min(njob, 65535), OB_THREADS, smem, s>>>(W, cc, gx, gw, tasks, jobs, njob, keep);
    MWG_CUDA(cudaGetLastError());
}

}  // namespace

void k_op_band(int K, const double *W, const double *cc, const double *gx, const double *gw, const OpBuildTask *tasks,
               int ntask, double *nrm, double *head, int *band, double *peak, double *keep, int nsm, cudaStream_t s) {
    if (ntask <= 0) return;
    switch (K) {
        case 4: launch_band<4>(W, cc, gx, gw, tasks, ntask, nrm, head, band, peak, keep, nsm, s); break;
        case 5: launch_band<5>(W, cc, gx, gw, tasks, ntask, nrm, head, band, peak, keep, nsm, s); break;
        case 6: launch_band<6>(W, cc, gx, gw, tasks, ntask, nrm, head, band, peak, keep, nsm, s); break;
        case 7: launch_band<7>(W, cc, gx, gw, tasks, ntask, nrm, head, band, peak, keep, nsm, s); break;
        case 8: launch_band<8>(W, cc, gx, gw, tasks, ntask, nrm, head, band, peak, keep, nsm, s); break;
        case 9: launch_band<9>(W, cc, gx, gw, tasks, ntask, nrm, head, band, peak, keep, nsm, s); break;
        case 10: launch_band<10>(W, cc, gx, gw, tasks, ntask, nrm, head, band, peak, keep, nsm, s); break;
        default: throw Error(MW_ERR_ARG, "no operator kernel for this order");
    }
}

void k_op_blocks(int K, const double *W, const double *cc, const double *gx, const double *gw, const OpBuildTask *tasks,
                 const OpBlockJob *jobs, int njob, const double *keep, cudaStream_t s) {
    if (njob <= 0) return;
    switch (K) {
        case 4: launch_blocks<4>(W, cc, gx, gw, tasks, jobs, njob, keep, s); break;
        case 5: launch_blocks<5>(W, cc, gx, gw, tasks, jobs, njob, keep, s); break;
        case 6: launch_blocks<6>(W, cc, gx, gw, tasks, jobs, njob, keep, s); break;
        case 7: launch_blocks<7>(W, cc, gx, gw, tasks, jobs, njob, keep, s); break;
        case 8: launch_blocks<8>(W, cc, gx, gw, tasks, jobs, njob, keep, s); break;
        case 9: launch_blocks<9>(W, cc, gx, gw, tasks, jobs, njob, keep, s); break;
        case 10: launch_blocks<10>(W, cc, gx, gw, tasks, jobs, njob, keep, s); break;
        default: throw Error(MW_ERR_ARG, "no operator kernel for this order");
    }
}

void k_op_convert(const double *blocks, float *b32, float *btc, float *btc2, long nblocks, int K, int NB, int groups,
                  cudaStream_t s) {
    if (nblocks <= 0) return;
    op_convert_kernel<<<1024, 256, 0, s>>>(blocks, b32, btc, btc2, nblocks, K, NB, groups);
    MWG_CUDA(cudaGetLastError());
}

}  // namespace mwg

// FP64 reduction kernels (Pauli expectations, norms), shared by the engine
// and the allocation-free entry point.
#pragma once
#include "device.cuh"
#include "kernels.h"

namespace qsv {

// ---------------------------------------------------------------------------
// FP64 reductions
// ---------------------------------------------------------------------------
template <int NT>
__device__ __forceinline__ double block_sum(double v, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0) {
        for (int i = 0; i < NT / 32; ++i) s += red[i];
    }
    return s;  // valid in thread 0
}

// v with its sign bit flipped where `neg` holds (integer work)
__device__ __forceinline__ double flip_sign(double v, unsigned neg) {
    return __hiloint2double(__double2hiint(v) ^ static_cast<int>(neg << 31), __double2loint(v));
}

// Amplitudes of one CTA step of the reductions below: element r of a thread is
// index base + threadIdx.x + 256 r, so index bits 8..10 are the thread's own,
// bits 0..7 the thread's and the others the step's.
constexpr int RED_ELEMS = 8;
constexpr uint64_t RED_STEP = 256 * RED_ELEMS;

// Z-only Pauli terms: sum_j |a_j|^2 (-1)^popcount(j & z_t)  (statevector.hpp:1281-1290).
// Bound by the FP64 pipe (2 instructions per clock and SM), so the terms share
// additions: a Walsh-Hadamard transform of the thread's 8 probabilities (24
// additions) gives every sign pattern of bits 8..10, of which each term adds
// one, signed by the parity of the other bits.  T terms cost 2 + 3 + T / 8 FP64
// instructions an amplitude instead of 2 + T (up to three terms are summed
// directly), and NB of them share one read of the state.
template <class P, int NB>
__global__ void __launch_bounds__(256) k_expect_z(const typename P::G* __restrict__ state, uint64_t N,
                                                  const uint64_t* __restrict__ zm, int nterms,
                                                  double* __restrict__ partial) {
    __shared__ double red[8];
    double acc[NB];
#pragma unroll
    for (int t = 0; t < NB; ++t) acc[t] = 0.0;
    for (uint64_t base = blockIdx.x * RED_STEP; base < N; base += gridDim.x * RED_STEP) {
        typename P::G g[RED_ELEMS];
        double h[RED_ELEMS];
#pragma unroll
        for (int r = 0; r < RED_ELEMS; ++r) {
            const uint64_t j = base + threadIdx.x + 256 * r;
            g[r] = j < N ? state[j] : P::make_g(0.0, 0.0);
        }
#pragma unroll
        for (int r = 0; r < RED_ELEMS; ++r) {
            const double re = P::gre(g[r]), im = P::gim(g[r]);
            h[r] = __fma_rn(re, re, __dmul_rn(im, im));
        }
        const uint64_t fixed = base | threadIdx.x;
        if (nterms > 3) {
#pragma unroll
            for (int b = 1; b < RED_ELEMS; b <<= 1)
#pragma unroll
                for (int r = 0; r < RED_ELEMS; ++r)
                    if (!(r & b)) {
                        const double u = h[r], v = h[r | b];
                        h[r] = u + v;
                        h[r | b] = u - v;
                    }
#pragma unroll
            for (int t = 0; t < NB; ++t)
                if (t < nterms) {
                    const uint64_t z = zm[t];
                    const int s = static_cast<int>(z >> 8) & 7;
                    const double a = (s & 1) ? ((s & 2) ? ((s & 4) ? h[7] : h[3]) : ((s & 4) ? h[5] : h[1]))
                                             : ((s & 2) ? ((s & 4) ? h[6] : h[2]) : ((s & 4) ? h[4] : h[0]));
                    acc[t] += flip_sign(a, __popcll(fixed & z) & 1);
                }
        } else {
#pragma unroll
            for (int t = 0; t < 3; ++t)
                if (t < nterms) {
                    const uint64_t z = zm[t];
                    const unsigned f = __popcll(fixed & z);
#pragma unroll
                    for (int r = 0; r < RED_ELEMS; ++r)
                        acc[t] += flip_sign(h[r], (f + __popc(r & static_cast<unsigned>(z >> 8))) & 1);
                }
        }
    }
#pragma unroll
    for (int t = 0; t < NB; ++t)
        if (t < nterms) {
            const double s = block_sum<256>(acc[t], red);
            if (threadIdx.x == 0) partial[static_cast<size_t>(blockIdx.x) * NB + t] = s;
        }
}

// Terms sharing one flip mask x: sum over pairs (i0, i0^x) of
// 2 Re(a_i0 conj(a_i1) phase) (statevector.hpp:1291-1304): terms with an even
// number of Y factors take the real part of a conj(b), the others the
// imaginary part.  A group of one term folds its sign into the operands and
// accumulates with two FP64 instructions a pair: bound by HBM then.
template <class P, int NB>
__global__ void __launch_bounds__(256) k_expect_x(const typename P::G* __restrict__ state, uint64_t N, uint64_t xmask,
                                                  int flip_q, const uint64_t* __restrict__ zm,
                                                  const int32_t* __restrict__ ny, int nterms,
                                                  double* __restrict__ partial) {
    constexpr int U = 4;  // pairs in flight per thread
    __shared__ double red[8];
    double acc[NB];
    bool even = false, odd = false;
#pragma unroll
    for (int t = 0; t < NB; ++t) {
        acc[t] = 0.0;
        if (t < nterms) {
            even |= (ny[t] & 1) == 0;
            odd |= (ny[t] & 1) != 0;
        }
    }
    const uint64_t half = N >> 1;
    for (uint64_t j0 = blockIdx.x * (256ULL * U) + threadIdx.x; j0 < half; j0 += gridDim.x * (256ULL * U)) {
        typename P::G ga[U], gb[U];
#pragma unroll
        for (int r = 0; r < U; ++r) {
            const uint64_t j = j0 + 256 * r;
            const uint64_t i0 = insert0(j, flip_q);
            ga[r] = j < half ? state[i0] : P::make_g(0.0, 0.0);
            gb[r] = j < half ? state[i0 ^ xmask] : P::make_g(0.0, 0.0);
        }
#pragma unroll
        for (int r = 0; r < U; ++r) {
            const uint64_t i0 = insert0(j0 + 256 * r, flip_q);
            const double ar = P::gre(ga[r]), ai = P::gim(ga[r]), br = P::gre(gb[r]), bi = P::gim(gb[r]);
            // v = a * conj(b); phase i^(2 parity + ny): vr, -vi, -vr, vi
            if (nterms == 1) {
                const int ph = ((__popcll(i0 & zm[0]) & 1) * 2 + ny[0]) & 3;
                const unsigned neg = ph == 1 || ph == 2;
                const double sr = flip_sign(ar, neg), si = flip_sign(ai, neg);
                acc[0] = even ? __fma_rn(sr, br, __fma_rn(si, bi, acc[0]))
                              : __fma_rn(si, br, __fma_rn(flip_sign(sr, 1), bi, acc[0]));
            } else {
                const double vr = even ? __fma_rn(ar, br, __dmul_rn(ai, bi)) : 0.0;
                const double vi = odd ? __fma_rn(ai, br, -__dmul_rn(ar, bi)) : 0.0;
#pragma unroll
                for (int t = 0; t < NB; ++t)
                    if (t < nterms) {
                        const int ph = ((__popcll(i0 & zm[t]) & 1) * 2 + ny[t]) & 3;
                        acc[t] += flip_sign((ph & 1) ? vi : vr, ph == 1 || ph == 2);
                    }
            }
        }
    }
#pragma unroll
    for (int t = 0; t < NB; ++t)
        if (t < nterms) {
            const double s = block_sum<256>(acc[t], red);
            if (threadIdx.x == 0) partial[static_cast<size_t>(blockIdx.x) * NB + t] = 2.0 * s;
        }
}

// out[t] = sum over the blocks of partial[b * stride + t]; CTA t
static __global__ void k_reduce_partials(const double* __restrict__ partial, int nblocks, int stride,
                                         double* __restrict__ out) {
    __shared__ double red[8];
    double s = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += 256) s += partial[static_cast<size_t>(b) * stride + blockIdx.x];
    s = block_sum<256>(s, red);
    if (threadIdx.x == 0) out[blockIdx.x] = s;
}

}  // namespace qsv

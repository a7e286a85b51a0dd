// Batched-run kernels.  A batch holds `items` states of n qubits back to back
// (item i at offset i << n) that share one plan; what differs per item is the
// coefficient pool (rewritten here from each item's slot values) and the
// results.  Every sum is FP64 and adds in a fixed order, so a batch run is
// deterministic and item i's result does not depend on the other items.
#include "kernels.h"
#include "reduce.cuh"

namespace qsv {

// Coefficients of a bindable gate at angle th, in the layout classify() uses
// for that gate (see bind_coef in plan.cpp).
__device__ __forceinline__ int bind_eval(int kind, double th, double* c) {
    double s, co;
    switch (kind) {
        case QFVM_OP_RX:
            sincos(0.5 * th, &s, &co);
            c[0] = co;
            c[1] = s;
            return 2;
        case QFVM_OP_RY:
            sincos(0.5 * th, &s, &co);
            c[0] = co;
            c[1] = -s;
            c[2] = s;
            c[3] = co;
            return 4;
        case QFVM_OP_RZ:
        case QFVM_OP_RZZ:
            sincos(0.5 * th, &s, &co);
            c[0] = co;
            c[1] = -s;
            c[2] = co;
            c[3] = s;
            return 4;
        case QFVM_OP_P:
        case QFVM_OP_CP:
            sincos(th, &s, &co);
            c[0] = 1.0;
            c[1] = 0.0;
            c[2] = co;
            c[3] = s;
            return 4;
        default: return 0;
    }
}

__device__ __forceinline__ void put_coef(double* d, double v) { *d = v; }
__device__ __forceinline__ void put_coef(float* d, double v) { *d = static_cast<float>(v); }
__device__ __forceinline__ void put_coef(ds* d, double v) {
    const float h = static_cast<float>(v);
    d->h = h;
    d->l = static_cast<float>(v - static_cast<double>(h));
}

// pool[item * cstride + bind.off ..] = coefficients at sign * vals[item * nslots + bind.slot]
template <class C>
__global__ void __launch_bounds__(256) k_bind(C* __restrict__ pool, uint64_t cstride, const Bind* __restrict__ binds,
                                              int nb, const double* __restrict__ vals, int nslots, int items) {
    const uint64_t total = static_cast<uint64_t>(items) * nb;
    for (uint64_t i = blockIdx.x * 256ULL + threadIdx.x; i < total; i += gridDim.x * 256ULL) {
        const uint64_t item = i / nb;
        const Bind bd = binds[i - item * nb];
        const double th = static_cast<double>(bd.sign) * vals[item * nslots + bd.slot];
        double c[4];
        const int m = bind_eval(bd.unit ? QFVM_OP_P : bd.kind, th, c);
        C* dst = pool + item * cstride + bd.off;
        for (int k = 0; k < m; ++k) put_coef(dst + k, c[k]);
    }
}

// pool[item * cstride + j] = pool[j] for items 1.. (the template is item 0)
template <class C>
__global__ void __launch_bounds__(256) k_replicate(C* __restrict__ pool, uint64_t cstride, uint64_t len, int items) {
    const uint64_t total = static_cast<uint64_t>(items - 1) * len;
    for (uint64_t i = blockIdx.x * 256ULL + threadIdx.x; i < total; i += gridDim.x * 256ULL) {
        const uint64_t item = 1 + i / len, j = i % len;
        pool[item * cstride + j] = pool[j];
    }
}

// amplitude 0 of every item = 1 (the rest was cleared by a memset)
template <class G>
__global__ void k_first_amp(G* __restrict__ state, int n, int items) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < items) {
        G one;
        one.x = 1;
        one.y = 0;
        state[static_cast<uint64_t>(i) << n] = one;
    }
}

// (P psi)[i] = i^ny (-1)^popcount((i ^ x) & z) psi[i ^ x]  (statevector.hpp:1281-1305).
// Both kernels below are bound by the FP64 pipe: a thread holds the RED_ELEMS
// indices that differ in bits 8..10 and shares its additions between terms as
// k_expect_z and k_hamiltonian do.

// Chunk sums of <psi|O_o|psi> for every observable o (terms optr[o]..optr[o+1],
// sorted by flip mask), FP64.  CTA c covers amplitudes [c * chunk, (c + 1) *
// chunk); chunk divides 2^n, so a chunk never spans items.  epart[c * nobs + o].
// NORM: also the chunk sums of |psi|^2, npart[c].
template <class P, bool NORM>
__global__ void __launch_bounds__(256) k_expect_seg(const typename P::G* __restrict__ psi, uint64_t chunk,
                                                    const uint64_t* __restrict__ xs, const uint64_t* __restrict__ zs,
                                                    const int32_t* __restrict__ ny, const double* __restrict__ cs,
                                                    const int32_t* __restrict__ optr, int nobs,
                                                    double* __restrict__ epart, double* __restrict__ npart) {
    __shared__ double red[8];
    const uint64_t lo = blockIdx.x * chunk, hi = lo + chunk;
    double nrm = 0.0;
    for (int o = 0; o < nobs; ++o) {
        const int t0 = optr[o], t1 = optr[o + 1];
        int td = t0;  // the terms without flips come first
        while (td < t1 && xs[td] == 0) ++td;
        double acc = 0.0;
        for (uint64_t base = lo; base < hi; base += RED_STEP) {
            const uint64_t fixed = base + threadIdx.x;  // base is a multiple of 2^11, or the item's start
            double re[RED_ELEMS], im[RED_ELEMS];
            {
                typename P::G g[RED_ELEMS];
#pragma unroll
                for (int r = 0; r < RED_ELEMS; ++r)
                    g[r] = fixed + 256 * r < hi ? psi[fixed + 256 * r] : P::make_g(0.0, 0.0);
#pragma unroll
                for (int r = 0; r < RED_ELEMS; ++r) {
                    re[r] = P::gre(g[r]);
                    im[r] = P::gim(g[r]);
                }
            }
            if (NORM && o == 0) {
#pragma unroll
                for (int r = 0; r < RED_ELEMS; ++r) nrm = __fma_rn(re[r], re[r], __fma_rn(im[r], im[r], nrm));
            }
            if (td == t0 + 1) {
                // one term: its signs go into the products
                const uint64_t z = zs[t0];
                const unsigned f = __popcll(fixed & z & ~0x700ULL);
                double s = 0.0;
#pragma unroll
                for (int r = 0; r < RED_ELEMS; ++r) {
                    const unsigned neg = (f + __popc((static_cast<unsigned>(fixed >> 8) + r) & static_cast<unsigned>(z >> 8) & 7u)) & 1;
                    s = __fma_rn(flip_sign(re[r], neg), re[r], __fma_rn(flip_sign(im[r], neg), im[r], s));
                }
                acc = __fma_rn(cs[t0], s, acc);
            } else if (td > t0) {
                double h[RED_ELEMS];
#pragma unroll
                for (int r = 0; r < RED_ELEMS; ++r) h[r] = __fma_rn(re[r], re[r], __dmul_rn(im[r], im[r]));
#pragma unroll
                for (int b = 1; b < RED_ELEMS; b <<= 1)
#pragma unroll
                    for (int r = 0; r < RED_ELEMS; ++r)
                        if (!(r & b)) {
                            const double u = h[r], v = h[r | b];
                            h[r] = u + v;
                            h[r | b] = u - v;
                        }
                for (int t = t0; t < td; ++t) {
                    const uint64_t z = zs[t];
                    const int s = static_cast<int>(z >> 8) & 7;
                    const double a = (s & 1) ? ((s & 2) ? ((s & 4) ? h[7] : h[3]) : ((s & 4) ? h[5] : h[1]))
                                             : ((s & 2) ? ((s & 4) ? h[6] : h[2]) : ((s & 4) ? h[4] : h[0]));
                    // element r is index fixed + 256 r: bits 8..10 of fixed are clear where the chunk has them
                    acc = __fma_rn(cs[t], flip_sign(a, __popcll(fixed & z) & 1), acc);
                }
            }
            uint64_t lastx = ~0ULL;
            double wr[RED_ELEMS], wi[RED_ELEMS];
            for (int t = td; t < t1; ++t) {
                const uint64_t x = xs[t], z = zs[t];
                if (x != lastx) {
#pragma unroll
                    for (int r = 0; r < RED_ELEMS; ++r) {
                        const typename P::G v = fixed + 256 * r < hi ? psi[(fixed + 256 * r) ^ x] : P::make_g(0.0, 0.0);
                        wr[r] = P::gre(v);
                        wi[r] = P::gim(v);
                    }
                    lastx = x;
                }
                const int y = ny[t] & 3;
                double s = 0.0;
#pragma unroll
                for (int r = 0; r < RED_ELEMS; ++r) {
                    // Re conj(p) i^y w, signed
                    const unsigned neg = (__popcll(((fixed + 256 * r) ^ x) & z) + (y >> 1)) & 1;
                    const double a = flip_sign(re[r], neg), b = flip_sign(im[r], neg);
                    s = (y & 1) ? __fma_rn(b, wr[r], __fma_rn(flip_sign(a, 1), wi[r], s))
                                : __fma_rn(a, wr[r], __fma_rn(b, wi[r], s));
                }
                acc = __fma_rn(cs[t], s, acc);
            }
        }
        const double s = block_sum<256>(acc, red);
        if (threadIdx.x == 0) epart[static_cast<uint64_t>(blockIdx.x) * nobs + o] = s;
    }
    if (NORM) {
        nrm = block_sum<256>(nrm, red);
        if (threadIdx.x == 0) npart[blockIdx.x] = nrm;
    }
}

// lam = sum_o w[item, o] O_o psi for every item (w == nullptr: all weights 1)
template <class P>
__global__ void __launch_bounds__(256) k_lambda_seg(const typename P::G* __restrict__ psi,
                                                    typename P::G* __restrict__ lam, uint64_t total, int n,
                                                    const uint64_t* __restrict__ xs, const uint64_t* __restrict__ zs,
                                                    const int32_t* __restrict__ ny, const double* __restrict__ cs,
                                                    const int32_t* __restrict__ tobs, int nterms, int nobs,
                                                    const double* __restrict__ w) {
    constexpr int U = 4;
    const uint64_t step = gridDim.x * 256ULL;
    // one term whose factor is a complex64 storage value: FP32 products round
    // as the FP64 product does when it is stored
    const bool one = sizeof(typename P::G) == 8 && nterms == 1 && !w &&
                     static_cast<double>(static_cast<float>(cs[0])) == cs[0];
    for (uint64_t i0 = blockIdx.x * 256ULL + threadIdx.x; i0 < total; i0 += step * U) {
        if (one) {
            const uint64_t x = xs[0], z = zs[0];
            const int y = ny[0] & 3;
            typename P::G v[U];
#pragma unroll
            for (int r = 0; r < U; ++r)
                v[r] = i0 + step * r < total ? psi[(i0 + step * r) ^ x] : P::make_g(0.0, 0.0);
#pragma unroll
            for (int r = 0; r < U; ++r) {
                const uint64_t i = i0 + step * r;
                if (i >= total) break;
                float c = static_cast<float>(cs[0]);
                if ((__popcll((i ^ x) & z) + (y >> 1)) & 1) c = -c;
                typename P::G o = v[r];
                o.x = static_cast<decltype(o.x)>((y & 1) ? -c * static_cast<float>(v[r].y) : c * static_cast<float>(v[r].x));
                o.y = static_cast<decltype(o.y)>((y & 1) ? c * static_cast<float>(v[r].x) : c * static_cast<float>(v[r].y));
                lam[i] = o;
            }
            continue;
        }
        double ar[U], ai[U], wr[U], wi[U];
#pragma unroll
        for (int r = 0; r < U; ++r) ar[r] = ai[r] = 0.0;
        uint64_t lastx = ~0ULL;
        for (int t = 0; t < nterms; ++t) {
            const uint64_t x = xs[t], z = zs[t];
            const int y = ny[t] & 3;
            if (x != lastx) {
#pragma unroll
                for (int r = 0; r < U; ++r) {
                    const uint64_t i = i0 + step * r;
                    const typename P::G v = i < total ? psi[i ^ x] : P::make_g(0.0, 0.0);
                    wr[r] = P::gre(v);
                    wi[r] = P::gim(v);
                }
                lastx = x;
            }
#pragma unroll
            for (int r = 0; r < U; ++r) {
                const uint64_t i = i0 + step * r;
                double c = cs[t];
                if (w && i < total) c *= w[(i >> n) * nobs + tobs[t]];
                c = flip_sign(c, (__popcll((i ^ x) & z) + (y >> 1)) & 1);
                if (y & 1) {
                    ar[r] = __fma_rn(flip_sign(c, 1), wi[r], ar[r]);
                    ai[r] = __fma_rn(c, wr[r], ai[r]);
                } else {
                    ar[r] = __fma_rn(c, wr[r], ar[r]);
                    ai[r] = __fma_rn(c, wi[r], ai[r]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < U; ++r) {
            const uint64_t i = i0 + step * r;
            if (i < total) lam[i] = P::make_g(ar[r], ai[r]);
        }
    }
}

// out[i * nobs + o] = sum_{k < per} in[(i * per + k) * nobs + o], divided by the
// item's sum of npart when there is one; inv[i] = 1 / that sum
__global__ void k_seg_sum(const double* __restrict__ in, int per, int segs, int nobs, double* __restrict__ out,
                          const double* __restrict__ npart, double* __restrict__ inv) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < segs * nobs) {
        const int seg = i / nobs, o = i - seg * nobs;
        double s = 0.0;
        for (int k = 0; k < per; ++k) s += in[(static_cast<size_t>(seg) * per + k) * nobs + o];
        if (npart) {
            double v = 0.0;
            for (int k = 0; k < per; ++k) v += npart[static_cast<size_t>(seg) * per + k];
            s /= v;
            if (o == 0) inv[seg] = 1.0 / v;
        }
        out[i] = s;
    }
}

// Per-item probe sums of a batched two-state pass: the item's tiles are
// consecutive, partial holds one row of ntiles values per probe.
__global__ void k_probe_reduce_seg(const double* __restrict__ partial, uint64_t ntiles, int tpi, int items, int np,
                                   double* __restrict__ out, int ostride, int ooff) {
    const uint64_t total = static_cast<uint64_t>(items) * np;
    for (uint64_t i = blockIdx.x * 256ULL + threadIdx.x; i < total; i += gridDim.x * 256ULL) {
        const uint64_t item = i / np;
        const int p = static_cast<int>(i - item * np);
        const double* src = partial + static_cast<uint64_t>(p) * ntiles + item * tpi;
        double s = 0.0;
        for (int t = 0; t < tpi; ++t) s += src[t];
        out[item * ostride + ooff + p] = s;
    }
}

// grads[item * nslots + s] = sum over the probes of slot s (ascending probe id)
__global__ void k_slot_gather(const double* __restrict__ vals, int nprobe, int items,
                              const int32_t* __restrict__ sptr, const int32_t* __restrict__ sidx, int nslots,
                              const double* __restrict__ inv, double* __restrict__ grads) {
    const uint64_t total = static_cast<uint64_t>(items) * nslots;
    for (uint64_t i = blockIdx.x * 256ULL + threadIdx.x; i < total; i += gridDim.x * 256ULL) {
        const uint64_t item = i / nslots;
        const int s = static_cast<int>(i - item * nslots);
        double g = 0.0;
        for (int k = sptr[s]; k < sptr[s + 1]; ++k) g += vals[item * nprobe + sidx[k]];
        grads[i] = inv ? g * inv[item] : g;
    }
}

static unsigned blocks_for(uint64_t work, unsigned cap = 152 * 8) {
    const uint64_t b = (work + 255) / 256;
    return static_cast<unsigned>(b < 1 ? 1 : (b < cap ? b : cap));
}

cudaError_t launch_bind(int arith, void* pool, uint64_t cstride, const Bind* dbinds, int nb, const double* dvals,
                        int nslots, int items, cudaStream_t st) {
    if (nb <= 0 || items <= 0) return cudaSuccess;
    const unsigned g = blocks_for(static_cast<uint64_t>(items) * nb);
    if (arith == QFVM_C64)
        k_bind<float><<<g, 256, 0, st>>>(static_cast<float*>(pool), cstride, dbinds, nb, dvals, nslots, items);
    else if (arith == QFVM_C128_DS)
        k_bind<ds><<<g, 256, 0, st>>>(static_cast<ds*>(pool), cstride, dbinds, nb, dvals, nslots, items);
    else
        k_bind<double><<<g, 256, 0, st>>>(static_cast<double*>(pool), cstride, dbinds, nb, dvals, nslots, items);
    return cudaGetLastError();
}

cudaError_t launch_replicate(int arith, void* pool, uint64_t cstride, uint64_t len, int items, cudaStream_t st) {
    if (items <= 1 || len == 0) return cudaSuccess;
    const unsigned g = blocks_for(static_cast<uint64_t>(items - 1) * len);
    if (arith == QFVM_C64)
        k_replicate<float><<<g, 256, 0, st>>>(static_cast<float*>(pool), cstride, len, items);
    else if (arith == QFVM_C128_DS)
        k_replicate<ds><<<g, 256, 0, st>>>(static_cast<ds*>(pool), cstride, len, items);
    else
        k_replicate<double><<<g, 256, 0, st>>>(static_cast<double*>(pool), cstride, len, items);
    return cudaGetLastError();
}

cudaError_t launch_zero_items(int storage, void* state, int n, int items, cudaStream_t st) {
    const size_t bytes = (static_cast<size_t>(items) << n) * (storage == QFVM_C64 ? 8 : 16);
    cudaError_t e = cudaMemsetAsync(state, 0, bytes, st);
    if (e != cudaSuccess) return e;
    const unsigned g = static_cast<unsigned>((items + 255) / 256);
    if (storage == QFVM_C64) k_first_amp<float2><<<g, 256, 0, st>>>(static_cast<float2*>(state), n, items);
    else k_first_amp<double2><<<g, 256, 0, st>>>(static_cast<double2*>(state), n, items);
    return cudaGetLastError();
}

// 32 amplitudes a thread: the reduction at the chunk's end costs ten FP64
// instructions a thread, an amplitude two to four
uint64_t hamiltonian_chunk(int n) { return n >= 13 ? 8192ULL : (1ULL << n); }

cudaError_t launch_expect_seg(int storage, const void* psi, int n, int items, const uint64_t* dx, const uint64_t* dz,
                              const int32_t* dny, const double* dc, const int32_t* doptr, int nobs, double* epart,
                              double* out, double* npart, double* inv, cudaStream_t st) {
    const uint64_t chunk = hamiltonian_chunk(n);
    const uint64_t per = (1ULL << n) / chunk;
    const uint64_t ctas = per * static_cast<uint64_t>(items);
    if (ctas > 0x7fffffffULL) return cudaErrorInvalidValue;
    if (storage == QFVM_C64 && npart)
        k_expect_seg<P32, true><<<static_cast<unsigned>(ctas), 256, 0, st>>>(
            static_cast<const float2*>(psi), chunk, dx, dz, dny, dc, doptr, nobs, epart, npart);
    else if (storage == QFVM_C64)
        k_expect_seg<P32, false><<<static_cast<unsigned>(ctas), 256, 0, st>>>(
            static_cast<const float2*>(psi), chunk, dx, dz, dny, dc, doptr, nobs, epart, nullptr);
    else
        k_expect_seg<P64, false><<<static_cast<unsigned>(ctas), 256, 0, st>>>(
            static_cast<const double2*>(psi), chunk, dx, dz, dny, dc, doptr, nobs, epart, nullptr);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const int outs = items * nobs;
    k_seg_sum<<<(outs + 127) / 128, 128, 0, st>>>(epart, static_cast<int>(per), items, nobs, out,
                                                storage == QFVM_C64 ? npart : nullptr, inv);
    return cudaGetLastError();
}

cudaError_t launch_lambda_seg(int storage, const void* psi, void* lam, int n, int items, const uint64_t* dx,
                              const uint64_t* dz, const int32_t* dny, const double* dc, const int32_t* dtobs,
                              int nterms, int nobs, const double* dw, cudaStream_t st) {
    const uint64_t total = static_cast<uint64_t>(items) << n;
    if (storage == QFVM_C64)
        k_lambda_seg<P32><<<blocks_for(total, 152 * 16), 256, 0, st>>>(static_cast<const float2*>(psi),
                                                                       static_cast<float2*>(lam), total, n, dx, dz,
                                                                       dny, dc, dtobs, nterms, nobs, dw);
    else
        k_lambda_seg<P64><<<blocks_for(total, 152 * 16), 256, 0, st>>>(static_cast<const double2*>(psi),
                                                                       static_cast<double2*>(lam), total, n, dx, dz,
                                                                       dny, dc, dtobs, nterms, nobs, dw);
    return cudaGetLastError();
}

cudaError_t launch_probe_reduce_seg(const double* partial, uint64_t ntiles, int tpi, int items, int np, double* out,
                                    int ostride, int ooff, cudaStream_t st) {
    if (np <= 0) return cudaSuccess;
    k_probe_reduce_seg<<<blocks_for(static_cast<uint64_t>(items) * np), 256, 0, st>>>(partial, ntiles, tpi, items, np,
                                                                                     out, ostride, ooff);
    return cudaGetLastError();
}

cudaError_t launch_slot_gather(const double* vals, int nprobe, int items, const int32_t* sptr, const int32_t* sidx,
                               int nslots, const double* inv, double* grads, cudaStream_t st) {
    if (nslots <= 0) return cudaSuccess;
    k_slot_gather<<<blocks_for(static_cast<uint64_t>(items) * nslots), 256, 0, st>>>(vals, nprobe, items, sptr, sidx,
                                                                                    nslots, inv, grads);
    return cudaGetLastError();
}

}  // namespace qsv

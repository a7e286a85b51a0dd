// Per-shot trajectories of circuits with mid-circuit measurement, reset and
// classically controlled blocks (the per-shot branch of qfvm.cpp:104-133).
// Shots run side by side as batch items (item i's state at i << n); every
// measure/reset is three kernels: FP64 outcome probabilities per item, the
// outcome drawn from the item's uniform, and the collapse (projection,
// 1/sqrt(p) scaling, and for reset the move of the outcome block to 0).
#include "kernels.h"
#include "reduce.cuh"

namespace qsv {

// index of group g (the 2^(n-k) assignments of the unmeasured qubits) with
// measured bits set to outcome m (bit j of m <-> qubit q[j]); srt = q sorted
__device__ __forceinline__ uint64_t group_index(uint64_t g, const uint8_t* srt, int k) {
    for (int j = 0; j < k; ++j) g = insert0(g, srt[j]);
    return g;
}
__device__ __forceinline__ uint64_t deposit(uint32_t m, const uint8_t* q, int k) {
    uint64_t d = 0;
    for (int j = 0; j < k; ++j)
        if ((m >> j) & 1) d |= 1ULL << q[j];
    return d;
}

// Measured qubits split at qubit 8: those below are bits of the thread index
// (256 consecutive amplitudes are read together whatever is measured), the
// others are stepped through.
struct MeasureSplit {
    uint32_t lo;       // mask of the measured qubits below 8
    int32_t kh;        // measured qubits above, their qubits ascending (srt) and by outcome bit (q)
    uint8_t srt[8], q[8], bit[8];  // bit: their place in the outcome
};
__device__ __forceinline__ uint32_t low_outcome(uint32_t t, const MeasureSpec& ms) {
    uint32_t m = 0;
    for (int j = 0; j < ms.k; ++j)
        if (ms.q[j] < 8) m |= ((t >> ms.q[j]) & 1u) << j;
    return m;
}

// part[(item * bpi + b) * 2^k + m] = sum over block b's amplitudes of outcome m
// of |a|^2: two FP64 instructions an amplitude, four amplitudes in flight a
// thread.  (Stepping through the outcomes of low qubits read every sector once
// per outcome: 5.0 ms for four of them on 2048 x 17 qubits, 1.0 ms now.)
template <class P>
__global__ void __launch_bounds__(256) k_outcome_probs(const typename P::G* __restrict__ state, int n, MeasureSpec ms,
                                                       MeasureSplit sp, uint64_t groups_per_block, int bpi,
                                                       double* __restrict__ part) {
    constexpr int U = 4;
    __shared__ double sums[8][32];
    const int item = blockIdx.x / bpi, b = blockIdx.x - item * bpi;
    const typename P::G* st = state + (static_cast<uint64_t>(item) << n);
    const uint64_t ng = 1ULL << (n - sp.kh);
    const uint64_t g0 = b * groups_per_block;
    const uint64_t g1 = g0 + groups_per_block < ng ? g0 + groups_per_block : ng;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t whi = sp.lo >> 5;  // measured bits of the warp index
    for (uint32_t mh = 0; mh < (1u << sp.kh); ++mh) {
        uint64_t dm = 0;
        uint32_t m = 0;
        for (int j = 0; j < sp.kh; ++j)
            if ((mh >> j) & 1) {
                dm |= 1ULL << sp.q[j];
                m |= 1u << sp.bit[j];
            }
        double acc[U];
#pragma unroll
        for (int r = 0; r < U; ++r) acc[r] = 0.0;
        for (uint64_t g = g0 + threadIdx.x; g < g1; g += 256 * U) {
            typename P::G a[U];
#pragma unroll
            for (int r = 0; r < U; ++r)
                a[r] = g + 256 * r < g1 ? st[group_index(g + 256 * r, sp.srt, sp.kh) | dm] : P::make_g(0.0, 0.0);
#pragma unroll
            for (int r = 0; r < U; ++r) {
                const double re = P::gre(a[r]), im = P::gim(a[r]);
                acc[r] = __fma_rn(re, re, __fma_rn(im, im, acc[r]));
            }
        }
        double s = (acc[0] + acc[1]) + (acc[2] + acc[3]);
        // over the unmeasured bits of the lane, then of the warp
#pragma unroll
        for (int o = 0; o < 5; ++o) {
            const double v = __shfl_xor_sync(0xffffffffu, s, 1 << o);
            if (!((sp.lo >> o) & 1)) s += v;
        }
        __syncthreads();
        sums[w][lane] = s;
        __syncthreads();
        if ((lane & ~sp.lo & 31u) == 0 && (w & ~whi & 7u) == 0) {
            double t = 0.0;
            for (uint32_t v = 0; v < 8; ++v)
                if ((v & whi) == static_cast<uint32_t>(w)) t += sums[v][lane];
            part[(static_cast<size_t>(blockIdx.x) << ms.k) + (m | low_outcome(threadIdx.x, ms))] = t;
        }
    }
}

// One thread per item: outcome probabilities (blocks summed in order), the
// first outcome m with u * total < cum[m], classical bits, scale 1/sqrt(p).
// istride: blocks of `part` from item to item (0: one state shared by all).
__global__ void k_outcome_choose(const double* __restrict__ part, int istride, int bpi, MeasureSpec ms, int items,
                                 const double* __restrict__ uni, int draw, int ndraws, uint8_t* __restrict__ creg,
                                 int ncb, int32_t* __restrict__ outcome, double* __restrict__ scale) {
    const int item = blockIdx.x * blockDim.x + threadIdx.x;
    if (item >= items) return;
    const uint32_t K = 1u << ms.k;
    double total = 0.0;
    for (uint32_t m = 0; m < K; ++m) {
        double p = 0.0;
        for (int b = 0; b < bpi; ++b) p = __dadd_rn(p, part[(static_cast<size_t>(item) * istride + b) * K + m]);
        total = __dadd_rn(total, p);
    }
    const double r = __dmul_rn(uni[static_cast<size_t>(item) * ndraws + draw], total);
    double cum = 0.0, pm = 0.0, plast = 0.0;
    uint32_t pick = K, last = 0;
    for (uint32_t m = 0; m < K; ++m) {
        double p = 0.0;
        for (int b = 0; b < bpi; ++b) p = __dadd_rn(p, part[(static_cast<size_t>(item) * istride + b) * K + m]);
        cum = __dadd_rn(cum, p);
        if (p > 0.0) {
            last = m;
            plast = p;
        }
        if (pick == K && r < cum) {
            pick = m;
            pm = p;
        }
    }
    if (pick == K) {
        pick = last;
        pm = plast;
    }
    outcome[item] = static_cast<int32_t>(pick);
    scale[item] = pm > 0.0 ? 1.0 / sqrt(pm) : 0.0;
    if (!ms.reset)
        for (int j = 0; j < ms.k; ++j) creg[static_cast<size_t>(item) * ncb + ms.cb[j]] = (pick >> j) & 1;
}

// Item by item, COLLAPSE_AMPS amplitudes a thread, two in flight: the amplitudes
// of the chosen outcome scaled, the others zero.  `src` is the item itself
// (a measure changes each amplitude in place) or one state shared by all items
// (sstride 0; then a reset reads its outcome's block for block 0).
constexpr int COLLAPSE_AMPS = 8;
template <class P>
__global__ void __launch_bounds__(256) k_collapse(const typename P::G* src, uint64_t sstride, typename P::G* state,
                                                  int n, MeasureSpec ms, int c_begin, int bpi,
                                                  const int32_t* __restrict__ outcome,
                                                  const double* __restrict__ scale) {
    const uint64_t item = c_begin + blockIdx.x / bpi;
    const uint64_t i0 = static_cast<uint64_t>(blockIdx.x % bpi) * (256 * COLLAPSE_AMPS) + threadIdx.x;
    const uint64_t N = 1ULL << n;
    const uint64_t all = deposit(~0u, ms.q, ms.k);
    const uint64_t from = deposit(static_cast<uint32_t>(outcome[item]), ms.q, ms.k);
    const uint64_t to = ms.reset ? 0 : from;
    const double sc = scale[item];
    const typename P::G* s = src + item * sstride;
    typename P::G* d = state + (item << n);
#pragma unroll 2
    for (int r = 0; r < COLLAPSE_AMPS; ++r) {
        const uint64_t i = i0 + 256 * r;
        if (i >= N) break;
        typename P::G v = P::make_g(0.0, 0.0);
        if ((i & all) == to) {
            const typename P::G a = s[(i & ~all) | from];
            v = P::make_g(sc * P::gre(a), sc * P::gim(a));
        }
        d[i] = v;
    }
}

// Reset in place: an item's outcome block, scaled, moves to block 0 and the
// rest is zeroed; one thread per group of the measured bits' values.
template <class P>
__global__ void __launch_bounds__(256) k_reset(typename P::G* __restrict__ state, int n, MeasureSpec ms, int c_begin,
                                               int items, const int32_t* __restrict__ outcome,
                                               const double* __restrict__ scale) {
    const int lg = n - ms.k;
    const uint64_t total = static_cast<uint64_t>(items - c_begin) << lg;
    for (uint64_t t = blockIdx.x * 256ULL + threadIdx.x; t < total; t += gridDim.x * 256ULL) {
        const uint64_t item = c_begin + (t >> lg);
        typename P::G* st = state + (item << n);
        const uint64_t base = group_index(t & ((1ULL << lg) - 1), ms.srt, ms.k);
        const double sc = scale[item];
        const typename P::G a = st[base | deposit(static_cast<uint32_t>(outcome[item]), ms.q, ms.k)];
        st[base] = P::make_g(sc * P::gre(a), sc * P::gim(a));
        for (uint32_t m = 1; m < (1u << ms.k); ++m) st[base | deposit(m, ms.q, ms.k)] = P::make_g(0.0, 0.0);
    }
}

// active[item] = (classical bits cb[0..nc) read as a binary number, first
// most significant) == condition   (check_cif, statevector.hpp:186-193)
__global__ void k_cif_mask(const uint8_t* __restrict__ creg, int ncb, int items, CifSpec cs,
                           uint8_t* __restrict__ active) {
    const int item = blockIdx.x * blockDim.x + threadIdx.x;
    if (item >= items) return;
    uint64_t v = 0;
    for (int j = 0; j < cs.nc; ++j) v = v * 2 + creg[static_cast<size_t>(item) * ncb + cs.cb[j]];
    active[item] = v == cs.condition ? 1 : 0;
}

// every item <- psi0 (2^n amplitudes, complex128 on the device)
__global__ void k_items_copy(double2* __restrict__ state, int n, int items, const double2* __restrict__ psi0) {
    const uint64_t N = 1ULL << n, total = N * static_cast<uint64_t>(items);
    for (uint64_t i = blockIdx.x * 256ULL + threadIdx.x; i < total; i += gridDim.x * 256ULL)
        state[i] = psi0[i & (N - 1)];
}

static unsigned grid_of(uint64_t work, unsigned cap = 152 * 16) {
    const uint64_t b = (work + 255) / 256;
    return static_cast<unsigned>(b < 1 ? 1 : (b < cap ? b : cap));
}

int outcome_blocks_per_item(int n, int k) {
    const uint64_t ng = 1ULL << (n - k);
    const uint64_t per = 256ULL * 16;  // groups per block
    return static_cast<int>((ng + per - 1) / per);
}

cudaError_t launch_measure(const void* shared, void* state, int n, const MeasureSpec& ms, int items, int c_begin,
                           const double* duni, int draw, int ndraws, uint8_t* dcreg, int ncb, double* dpart,
                           int32_t* doutcome, double* dscale, cudaStream_t st) {
    MeasureSplit sp{};
    for (int j = 0; j < ms.k; ++j) {
        if (ms.q[j] < 8) {
            sp.lo |= 1u << ms.q[j];
        } else {
            sp.q[sp.kh] = ms.q[j];
            sp.bit[sp.kh++] = static_cast<uint8_t>(j);
        }
    }
    for (int j = 0, h = 0; j < ms.k; ++j)
        if (ms.srt[j] >= 8) sp.srt[h++] = ms.srt[j];
    const int bpi = outcome_blocks_per_item(n, ms.k);
    const uint64_t gpb = (256ULL * 16) << (ms.k - sp.kh);  // the same blocks however the outcome splits
    const double2* src = static_cast<const double2*>(shared ? shared : state);
    k_outcome_probs<P64><<<static_cast<unsigned>(bpi) * (shared ? 1 : items), 256, 0, st>>>(src, n, ms, sp, gpb, bpi,
                                                                                            dpart);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_outcome_choose<<<(items + 127) / 128, 128, 0, st>>>(dpart, shared ? 0 : bpi, bpi, ms, items, duni, draw, ndraws,
                                                          dcreg, ncb, doutcome, dscale);
    e = cudaGetLastError();
    if (e != cudaSuccess || c_begin >= items) return e;
    if (ms.reset && !shared) {
        k_reset<P64><<<grid_of(static_cast<uint64_t>(items - c_begin) << (n - ms.k)), 256, 0, st>>>(
            static_cast<double2*>(state), n, ms, c_begin, items, doutcome, dscale);
    } else {
        const uint64_t per = 256ULL * COLLAPSE_AMPS;
        const int cpi = static_cast<int>(((1ULL << n) + per - 1) / per);
        k_collapse<P64><<<static_cast<unsigned>(cpi) * (items - c_begin), 256, 0, st>>>(
            src, shared ? 0 : 1ULL << n, static_cast<double2*>(state), n, ms, c_begin, cpi, doutcome, dscale);
    }
    return cudaGetLastError();
}

cudaError_t launch_cif_mask(const uint8_t* dcreg, int ncb, int items, const CifSpec& cs, uint8_t* dactive,
                            cudaStream_t st) {
    k_cif_mask<<<(items + 127) / 128, 128, 0, st>>>(dcreg, ncb, items, cs, dactive);
    return cudaGetLastError();
}

cudaError_t launch_items_copy(void* state, int n, int items, const void* psi0, cudaStream_t st) {
    k_items_copy<<<grid_of((1ULL << n) * items), 256, 0, st>>>(static_cast<double2*>(state), n, items,
                                                              static_cast<const double2*>(psi0));
    return cudaGetLastError();
}

}  // namespace qsv

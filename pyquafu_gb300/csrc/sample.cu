// Exact shot sampling in parallel.
//
// The reference draws a shot by scanning the state in index order with an
// FP64 running sum, p = fl(p + q_i), q_i = fl(fl(re^2) + fl(im^2)), and
// returning the first i with r < p (N when there is none;
// statevector.hpp:1380-1412).  That sum is sequential, but its rounding has
// structure: while p stays inside one binade [2^e, 2^(e+1)), p is a multiple
// of G = 2^(e-52) and fl(p + q) = p + G * round(q / G), the rounding of q
// alone onto the grid G (independent of p), except for exact ties, whose
// round-half-even direction depends on p's last bit.  So:
//
//   1. k_approx_sums, k_approx_scan: FP32 sums of |a|^2 over blocks of
//      SAMPLE_BS elements and their prefix.  They only say in which binade
//      (or two) each block's running sum can lie.
//   2. k_block_counts (all SMs): per block and candidate binade the saturating
//      sum of round(q_i / G) and whether a tie occurs.
//   3. k_exact_scan (one CTA): the exact running sum at every block start.
//      Up to 1024 blocks that stay inside the current binade and have no tie
//      advance it by one integer prefix sum.  A block that crosses a binade,
//      holds a tie or was given other candidates is resolved by the whole CTA
//      in the same way at 4 elements a thread: integer prefix sums between
//      its events, the reference's own FP64 additions on the 4 elements around
//      each event.
//   4. k_sample_shots (a warp per shot): binary search of the block whose exact
//      end exceeds r, then inside the block integer prefix sums against r on
//      the grid, or, in a resolved block, the recorded running sums.
//
// Every value is the reference's own FP64 running sum, so every sampled index
// equals the sequential scan's, with no uncertain case left.  All loops are
// bounded by the state length.
//
// Bounds and figures (28 qubits complex128, 4096 shots): step 1 reads the state
// at the copy bandwidth; step 2 is bound by the three FP64 instructions that
// form q (2 per clock and SM); steps 3 and 4 are latency.  Counting 16 candidate
// binades per element, walking 32 blocks a step on one warp and adding the
// elements of a shot's block one by one took 19.7 ms for what takes 2.9 ms now.
#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.h"
#include "policy.cuh"

namespace qsv {

namespace {

constexpr uint64_t KCAP = 1ULL << 60;  // saturation of grid counts (any binade has < 2^53 steps)
constexpr uint64_t MTOP = 1ULL << 53;  // a binade's grid has 2^52 .. 2^53 - 1 steps from 0
constexpr int E_LOW = -1022;           // lowest binade: its grid is the subnormals' as well
constexpr int PER = SAMPLE_BS / 1024;  // elements per thread of a resolved block
constexpr int MAX_EVENTS = 64;         // events of a resolved block before it is summed element by element

template <class P>
__device__ __forceinline__ double qprob(const typename P::G g) {
    const double re = P::gre(g), im = P::gim(g);
    return __dadd_rn(__dmul_rn(re, re), __dmul_rn(im, im));
}

__device__ __forceinline__ uint64_t sat_add(uint64_t a, uint64_t b) {
    const uint64_t s = a + b;  // a, b <= KCAP: no wrap
    return s > KCAP ? KCAP : s;
}

// round(q / 2^(e-52)) for q >= 0 (nearest; *tie when q sits exactly half-way)
__device__ __forceinline__ uint64_t grid_count(double q, int e, bool* tie) {
    const uint64_t bits = static_cast<uint64_t>(__double_as_longlong(q));
    const int ex = static_cast<int>((bits >> 52) & 0x7FF);
    uint64_t mant = bits & ((1ULL << 52) - 1);
    int eb = 1;
    if (ex != 0) {
        mant |= 1ULL << 52;
        eb = ex;
    }
    *tie = false;
    if (mant == 0) return 0;
    const int sh = eb - 1023 - e;  // q / G = mant * 2^sh
    if (sh >= 0) return sh >= 7 ? KCAP : (mant << sh);
    const int d = -sh;
    if (d > 54) return 0;  // q < G / 4
    const uint64_t qi = mant >> d;
    const uint64_t rem = mant & ((1ULL << d) - 1);
    const uint64_t half = 1ULL << (d - 1);
    *tie = rem == half;
    return qi + (rem > half ? 1 : 0);
}

__device__ __forceinline__ int binade_of(double p) {  // p >= 0; zero and subnormals join the lowest binade
    const int e = static_cast<int>((static_cast<uint64_t>(__double_as_longlong(p)) >> 52) & 0x7FF) - 1023;
    return e < E_LOW ? E_LOW : e;
}
// p = m * 2^(e - 52), exactly (p finite, in binade e)
__device__ __forceinline__ uint64_t steps_of(double p, int e) {
    const uint64_t bits = static_cast<uint64_t>(__double_as_longlong(p));
    const uint64_t mant = bits & ((1ULL << 52) - 1);
    return ((bits >> 52) & 0x7FF) ? (mant | (1ULL << 52)) : (e == E_LOW ? mant : 0);
}
__device__ __forceinline__ double value_of(uint64_t m, int e) {  // m < 2^53, and m >= 2^52 unless e is the lowest
    return m < (1ULL << 52) ? __longlong_as_double(static_cast<long long>(m))
                            : __longlong_as_double(static_cast<long long>(
                                  (m & ((1ULL << 52) - 1)) | (static_cast<uint64_t>(e + 1023) << 52)));
}

// an amplitude's |a|^2 to FP32 accuracy, no FP64 instruction (a double's high
// word carries its exponent and 20 mantissa bits)
__device__ __forceinline__ float trunc_float(double v) {
    const uint32_t hw = static_cast<uint32_t>(__double2hiint(v)) & 0x7FFFFFFFu, lw = static_cast<uint32_t>(__double2loint(v));
    const uint32_t f = __funnelshift_l(lw, hw, 3) - 0xC0000000u;  // FP32 exponent = FP64 exponent - 896
    return hw < 0x38200000u ? 0.f : (hw >= 0x47E00000u ? __int_as_float(0x7F800000) : __uint_as_float(f));
}
__device__ __forceinline__ float approx_prob(double2 g) {
    const float x = trunc_float(g.x), y = trunc_float(g.y);
    return fmaf(x, x, y * y);
}
__device__ __forceinline__ float approx_prob(float2 g) { return fmaf(g.x, g.x, g.y * g.y); }

template <class G>
__global__ void __launch_bounds__(256) k_approx_sums(const G* __restrict__ state, uint64_t N, uint64_t nb,
                                                     float* __restrict__ bsum) {
    __shared__ float red[8];
    for (uint64_t b = blockIdx.x; b < nb; b += gridDim.x) {
        const uint64_t i0 = b * SAMPLE_BS + threadIdx.x;
        float s = 0.f;
#pragma unroll
        for (int r = 0; r < SAMPLE_BS / 256; ++r) {
            const uint64_t i = i0 + 256 * r;
            if (i < N) s += approx_prob(state[i]);
        }
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
        __syncthreads();
        if (threadIdx.x == 0) {
            float t = 0.f;
            for (int w = 0; w < 8; ++w) t += red[w];
            bsum[b] = t;
        }
        __syncthreads();
    }
}

// Exclusive prefix of the block sums (one CTA, 8 blocks a thread and step);
// pre[nb] = total.
__global__ void __launch_bounds__(1024) k_approx_scan(const float* __restrict__ bsum, uint64_t nb,
                                                      double* __restrict__ pre) {
    constexpr int V = 8;
    __shared__ double wsum[32];
    __shared__ double carry;
    if (threadIdx.x == 0) carry = 0.0;
    __syncthreads();
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (uint64_t base = 0; base < nb; base += 1024 * V) {
        const uint64_t i0 = base + static_cast<uint64_t>(threadIdx.x) * V;
        float v[V], run[V];  // the sums of one thread to FP32
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < V; ++k) v[k] = i0 + k < nb ? bsum[i0 + k] : 0.f;
#pragma unroll
        for (int k = 0; k < V; ++k) {
            run[k] = s;
            s += v[k];
        }
        double x = s;
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, x, o);
            if (l >= o) x += y;
        }
        if (l == 31) wsum[w] = x;
        __syncthreads();
        if (w == 0) {
            double z = wsum[l];
            for (int o = 1; o < 32; o <<= 1) {
                const double y = __shfl_up_sync(0xffffffffu, z, o);
                if (l >= o) z += y;
            }
            wsum[l] = z;
        }
        __syncthreads();
        const double before = carry + (w > 0 ? wsum[w - 1] : 0.0) + (x - s);
#pragma unroll
        for (int k = 0; k < V; ++k)
            if (i0 + k < nb) pre[i0 + k] = before + run[k];
        __syncthreads();
        if (threadIdx.x == 1023) carry += wsum[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) pre[nb] = carry;
}

// Grid counts of every block at the binade its approximate start lies in and,
// where the approximate sums allow for it, at the next one.
template <class P>
__global__ void __launch_bounds__(256) k_block_counts(const typename P::G* __restrict__ state, uint64_t N, uint64_t nb,
                                                      const double* __restrict__ pre, SampleBlock* __restrict__ blk) {
    __shared__ uint64_t red[8];
    __shared__ int tred[8];
    constexpr double SLACK = 1.0 / (1 << 16);  // the approximate sums are good to about 2^-20
    for (uint64_t b = blockIdx.x; b < nb; b += gridDim.x) {
        const int e0 = binade_of(pre[b] * (1.0 - SLACK));
        const int e1 = binade_of(pre[b + 1] * (1.0 + SLACK));
        const uint64_t i0 = b * SAMPLE_BS + threadIdx.x;
        for (int c = 0; c < (e1 > e0 ? 2 : 1); ++c) {
            uint64_t acc = 0;
            bool tie = false;
#pragma unroll 8
            for (int r = 0; r < SAMPLE_BS / 256; ++r) {
                const uint64_t i = i0 + 256 * r;
                if (i < N) {
                    bool t;
                    acc = sat_add(acc, grid_count(qprob<P>(state[i]), e0 + c, &t));
                    tie |= t;
                }
            }
            for (int o = 16; o; o >>= 1) acc = sat_add(acc, __shfl_xor_sync(0xffffffffu, acc, o));
            const int any = __any_sync(0xffffffffu, tie);
            if ((threadIdx.x & 31) == 0) {
                red[threadIdx.x >> 5] = acc;
                tred[threadIdx.x >> 5] = any;
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                uint64_t v = 0;
                int t = 0;
                for (int w = 0; w < 8; ++w) {
                    v = sat_add(v, red[w]);
                    t |= tred[w];
                }
                blk[b].cnt[c] = t ? KCAP : v;  // a tie: as a crossing, resolved by the scan
                if (c == 0) blk[b].e = e0;
                if (c == 0) blk[b].two = e1 > e0;
            }
            __syncthreads();
        }
    }
}

// Saturating inclusive prefix over the CTA's 1024 threads.
__device__ __forceinline__ uint64_t cta_prefix(uint64_t v, uint64_t* wtot) {
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(0xffffffffu, v, o);
        if (l >= o) v = sat_add(v, y);
    }
    if (l == 31) wtot[w] = v;
    __syncthreads();
    if (w == 0) {
        uint64_t z = wtot[l];
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t y = __shfl_up_sync(0xffffffffu, z, o);
            if (l >= o) z = sat_add(z, y);
        }
        wtot[l] = z;
    }
    __syncthreads();
    const uint64_t r = w > 0 ? sat_add(v, wtot[w - 1]) : v;
    __syncthreads();
    return r;
}
// index of the first thread with bad set (1024: none)
__device__ __forceinline__ int cta_first(bool bad, int* first) {
    if (threadIdx.x == 0) *first = 1024;
    __syncthreads();
    const unsigned m = __ballot_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0 && m) atomicMin(first, static_cast<int>(threadIdx.x) + __ffs(m) - 1);
    __syncthreads();
    const int f = *first;
    __syncthreads();
    return f;
}

// One CTA: start[b], the exact running sum at every block start (start[nb]:
// over the whole state).  slot[b]: -1 for a block advanced by its count, else
// the place of its running sums in `fine` (one per PER elements), or -2 when
// all SAMPLE_SLOTS places are taken.  *seq counts the blocks resolved here.
template <class P>
__global__ void __launch_bounds__(1024) k_exact_scan(const typename P::G* __restrict__ state, uint64_t N, uint64_t nb,
                                                     const SampleBlock* __restrict__ blk, double* __restrict__ start,
                                                     int32_t* __restrict__ slot, double* __restrict__ fine,
                                                     int64_t* __restrict__ seq) {
    __shared__ uint64_t wtot[32];
    __shared__ int first_s;
    __shared__ double p_s;
    __shared__ double qs[SAMPLE_BS];
    const int tid = threadIdx.x;
    double p = 0.0;
    int64_t nres = 0;
    uint64_t b = 0;
    while (b < nb) {
        const bool finite = p < __longlong_as_double(0x7FF0000000000000LL);  // false for infinity and NaN
        if (finite) {
            const int e = binade_of(p);
            const uint64_t m = steps_of(p, e);
            const uint64_t i = b + tid;
            uint64_t k = KCAP;
            if (i < nb) {
                const SampleBlock v = blk[i];
                if (v.e == e) k = v.cnt[0];
                else if (v.two && v.e + 1 == e) k = v.cnt[1];
            }
            const uint64_t incl = cta_prefix(k, wtot);
            const bool ok = k < KCAP && m + incl < MTOP;  // the block ends inside the binade
            const int f = cta_first(!ok, &first_s);
            if (tid < f) {
                start[i] = value_of(m + incl - k, e);
                slot[i] = -1;
            }
            if (f > 0 && tid == f - 1) p_s = value_of(m + incl, e);
            __syncthreads();
            if (f > 0) p = p_s;
            __syncthreads();
            b += f;
            if (f == 1024 || b >= nb) continue;
        }
        // block b: PER elements a thread
        const uint64_t i0 = b * SAMPLE_BS + static_cast<uint64_t>(tid) * PER;
        double q[PER];
#pragma unroll
        for (int r = 0; r < PER; ++r) {
            q[r] = i0 + r < N ? qprob<P>(state[i0 + r]) : 0.0;
            qs[tid * PER + r] = q[r];
        }
        const int place = nres < SAMPLE_SLOTS ? static_cast<int>(nres) : -2;
        double* fo = place >= 0 ? fine + static_cast<size_t>(place) * 1024 : nullptr;
        ++nres;
        if (tid == 0) {
            start[b] = p;
            slot[b] = place;
        }
        __syncthreads();
        int cur = 0;
        for (int ev = 0; cur < 1024; ++ev) {
            if (ev == MAX_EVENTS || !(p < __longlong_as_double(0x7FF0000000000000LL))) {
                if (tid == 0) {
                    double s = p;
                    for (int t = cur; t < 1024; ++t) {
                        if (fo) fo[t] = s;
                        for (int r = 0; r < PER; ++r) s = __dadd_rn(s, qs[t * PER + r]);
                    }
                    p_s = s;
                }
                __syncthreads();
                p = p_s;
                __syncthreads();
                break;
            }
            const int e = binade_of(p);
            const uint64_t m = steps_of(p, e);
            uint64_t k = 0;
            bool tie = false;
            if (tid >= cur) {
#pragma unroll
                for (int r = 0; r < PER; ++r) {
                    bool t;
                    k = sat_add(k, grid_count(q[r], e, &t));
                    tie |= t;
                }
                if (k > 2 * MTOP) k = 2 * MTOP;  // past any binade; keeps the first event's prefix unsaturated
            }
            const uint64_t incl = cta_prefix(k, wtot);
            const int f = cta_first(tid >= cur && (tie || m + incl >= MTOP), &first_s);
            if (tid >= cur && tid < f && fo) fo[tid] = value_of(m + incl - k, e);
            if (f == 1024) {
                if (tid == 1023) p_s = value_of(m + incl, e);
            } else if (tid == f) {
                double s = value_of(m + incl - k, e);  // before this thread's elements: still inside the binade
                if (fo) fo[tid] = s;
#pragma unroll
                for (int r = 0; r < PER; ++r) s = __dadd_rn(s, q[r]);
                p_s = s;
            }
            __syncthreads();
            p = p_s;
            __syncthreads();
            cur = f == 1024 ? 1024 : f + 1;
        }
        ++b;
    }
    if (tid == 0) {
        start[nb] = p;
        *seq = nres;
    }
}

// A warp per shot: the first index whose running sum exceeds r.
template <class P>
__global__ void __launch_bounds__(256) k_sample_shots(const typename P::G* __restrict__ state, uint64_t N,
                                                      uint64_t nb, const double* __restrict__ start,
                                                      const int32_t* __restrict__ slot,
                                                      const double* __restrict__ fine,
                                                      const double* __restrict__ uni, int64_t shots,
                                                      uint64_t* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t s = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (s >= shots) return;
    const double r = uni[s];
    if (!(r < start[nb])) {
        if (lane == 0) out[s] = N;
        return;
    }
    // first block with r < start[b + 1]
    uint64_t lo = 0, hi = nb - 1;
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if (r < start[mid + 1]) hi = mid;
        else lo = mid + 1;
    }
    const int place = slot[lo];
    const uint64_t i0 = lo * SAMPLE_BS, i1 = (i0 + SAMPLE_BS < N) ? i0 + SAMPLE_BS : N;
    uint64_t found = i1 - 1;  // start[lo + 1] > r: the block's last index at the latest
    if (place >= 0) {
        // the thread of the scan whose elements pass r, then its elements
        const double* f = fine + static_cast<size_t>(place) * 1024;
        int a = 0, z = 1023;
        while (a < z) {
            const int mid = (a + z) >> 1;
            if (r < f[mid + 1]) z = mid;
            else a = mid + 1;
        }
        double p = f[a];
        for (int j = 0; j < PER; ++j) {
            const uint64_t i = i0 + static_cast<uint64_t>(a) * PER + j;
            if (i >= i1) break;
            p = __dadd_rn(p, qprob<P>(state[i]));
            if (r < p) {
                found = i;
                break;
            }
        }
    } else if (place == -1) {
        // running sums m + K_i on the block's grid: the first K_i with m + K_i > r / G
        const double p = start[lo];
        const int e = binade_of(p);
        const uint64_t m = steps_of(p, e);
        const double x = e == E_LOW ? ldexp(ldexp(r, 1022), 52) : ldexp(r, 52 - e);  // exact: r < 2^(e+1)
        const uint64_t need = r < p ? 0 : static_cast<uint64_t>(x) + 1 - m;  // (r < p: a negative r in block 0)
        uint64_t acc = 0;
        for (uint64_t i = i0 + lane * PER; i - lane * PER < i1; i += 32 * PER) {
            uint64_t k[PER], sum = 0;
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                bool t;
                sum += i + j < i1 ? grid_count(qprob<P>(state[i + j]), e, &t) : 0;
                k[j] = sum;
            }
            uint64_t incl = sum;
            for (int o = 1; o < 32; o <<= 1) {
                const uint64_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const unsigned hit = __ballot_sync(0xffffffffu, acc + incl >= need);
            if (hit) {
                const int src = __ffs(hit) - 1;
                uint64_t at = i + PER - 1;
#pragma unroll
                for (int j = PER - 1; j >= 0; --j)
                    if (acc + incl - sum + k[j] >= need) at = i + j;
                found = __shfl_sync(0xffffffffu, at, src);
                break;
            }
            acc += __shfl_sync(0xffffffffu, incl, 31);
        }
    } else {
        double p = start[lo];
        bool done = false;
        for (uint64_t i = i0; i < i1 && !done; i += 32) {
            const double q = (i + lane < i1) ? qprob<P>(state[i + lane]) : 0.0;
            for (int j = 0; j < 32 && i + j < i1; ++j) {
                p = __dadd_rn(p, __shfl_sync(0xffffffffu, q, j));
                if (r < p) {
                    found = i + j;
                    done = true;
                    break;
                }
            }
        }
    }
    if (lane == 0) out[s] = found;
}

template <class P>
cudaError_t launch_all(const void* state, uint64_t N, const SampleScratch& w, const double* uni, int64_t shots,
                       uint64_t* out, cudaStream_t st) {
    using G = typename P::G;
    const G* s = static_cast<const G*>(state);
    const uint64_t nb = (N + SAMPLE_BS - 1) / SAMPLE_BS;
    const unsigned g1 = static_cast<unsigned>(nb < 152 * 8 ? nb : 152 * 8);
    k_approx_sums<G><<<g1, 256, 0, st>>>(s, N, nb, w.bsum);
    k_approx_scan<<<1, 1024, 0, st>>>(w.bsum, nb, w.pre);
    k_block_counts<P><<<g1, 256, 0, st>>>(s, N, nb, w.pre, w.blk);
    k_exact_scan<P><<<1, 1024, 0, st>>>(s, N, nb, w.blk, w.start, w.slot, w.fine, w.seq);
    const unsigned g3 = static_cast<unsigned>((static_cast<uint64_t>(shots) * 32 + 255) / 256);
    k_sample_shots<P><<<g3, 256, 0, st>>>(s, N, nb, w.start, w.slot, w.fine, uni, shots, out);
    return cudaGetLastError();
}

}  // namespace

size_t sample_scratch_bytes(uint64_t N) {
    SampleScratch w;
    return sample_scratch(N, nullptr, &w);
}

size_t sample_scratch(uint64_t N, void* base, SampleScratch* w) {
    const uint64_t nb = (N + SAMPLE_BS - 1) / SAMPLE_BS;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* p = static_cast<char*>(base) + off;
        off += (bytes + 255) / 256 * 256;
        return static_cast<void*>(p);
    };
    w->bsum = static_cast<float*>(take(nb * sizeof(float)));
    w->pre = static_cast<double*>(take((nb + 1) * sizeof(double)));
    w->blk = static_cast<SampleBlock*>(take(nb * sizeof(SampleBlock)));
    w->start = static_cast<double*>(take((nb + 1) * sizeof(double)));
    w->slot = static_cast<int32_t*>(take(nb * sizeof(int32_t)));
    w->fine = static_cast<double*>(take(static_cast<size_t>(SAMPLE_SLOTS) * 1024 * sizeof(double)));
    w->seq = static_cast<int64_t*>(take(sizeof(int64_t)));
    return off;
}

cudaError_t launch_sample(int precision, const void* state, uint64_t N, const SampleScratch& w, const double* uni,
                          int64_t shots, uint64_t* out, cudaStream_t st) {
    if (precision == QFVM_C64) return launch_all<P32>(state, N, w, uni, shots, out, st);
    return launch_all<P64>(state, N, w, uni, shots, out, st);
}

}  // namespace qsv

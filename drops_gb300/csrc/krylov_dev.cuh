// Device building blocks of the persistent Krylov kernels: bounded grid
// barriers, fixed-order reductions, the scalar state of a solve and the
// SELL row product.
#pragma once
#include "ff.cuh"
#include "tf_internal.cuh"

namespace tf {

constexpr int kKryThreads = 256;

// Loads of vectors that the same persistent launch writes (basis vectors,
// search directions, iterates) and reads again after a grid barrier.  They go
// through L1 (ld.global.ca): neighbouring rows gather largely the same
// entries, and an 8-byte gather that misses L1 costs a whole 32-byte L2
// sector.  Every such read happens after the barrier of the step that wrote
// the data, i.e. after thread 0's fence following the release it observed and
// the block's bar.sync, which orders it after the writes in the memory model.
template <class T>
__device__ __forceinline__ T kld(const T* p) { return __ldca(p); }

// ---------------------------------------------------------------------------
// grid barrier with a bounded wait
// ---------------------------------------------------------------------------
struct GridSync {
    unsigned* count;
    unsigned* gen;
    int* status;
};
constexpr long long kSpinLimit = 20000000;  // ~1-2 s with the backoff below

__device__ __forceinline__ bool grid_barrier(const GridSync& g) {
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile unsigned* vgen = g.gen;
        const unsigned my = *vgen;
        __threadfence();
        if (atomicAdd(g.count, 1u) == gridDim.x - 1) {
            *g.count = 0;
            __threadfence();
            atomicAdd(g.gen, 1u);
        } else {
            long long spins = 0;
            while (*vgen == my) {
                if (++spins > kSpinLimit) {
                    atomicCAS(g.status, 0, TF_ERR_WATCHDOG);
                    break;
                }
                if (spins > 256) __nanosleep(32);
            }
        }
        __threadfence();
    }
    __syncthreads();
    __shared__ int st;
    if (threadIdx.x == 0) st = *((volatile int*)g.status);
    __syncthreads();
    return st == 0;
}

// ---------------------------------------------------------------------------
// reductions: warp xor-trees (every lane ends with the same sum), one FP64
// partial per block, and a fixed-order sum of all partials in every block
// ---------------------------------------------------------------------------
template <class T>
__device__ __forceinline__ T warp_sum(T v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums of doubles in fixed point.  An FP64 add holds a quarter of the SM's
// FP64 pipe for 64 cycles on GB300 whatever the number of active lanes (a
// chain of adds costs 66 cycles each, measured), so a butterfly or a serial sum
// of partials is a chain of hundreds of cycles.  Here every mantissa is aligned
// to the largest exponent of the sum (rounded to nearest, at 2^-2 to 2^-9 ulp of
// the largest value) and the integers are added: a sum in any order gives the
// same bits, about 15 integer instructions per value and one FP64-pipe
// instruction per result (the conversion back, the only rounding to 53 bits).
struct FxTerm {
    unsigned e;            // biased exponent, 1 for subnormals and zero
    unsigned long long m;  // mantissa with the hidden bit
    bool neg;
};
__device__ __forceinline__ FxTerm fx_term(double v) {
    const long long b = __double_as_longlong(v);
    const unsigned e = (unsigned)(b >> 52) & 0x7ffu;
    FxTerm t;
    t.e = max(e, 1u);
    t.m = ((unsigned long long)b & 0xfffffffffffffull) | (e ? 1ull << 52 : 0ull);
    t.neg = b < 0;
    return t;
}
// the term in units of 2^(emax - 1075 - left)
__device__ __forceinline__ long long fx_align(const FxTerm& t, unsigned emax, int left) {
    const unsigned sh = emax - t.e;
    const unsigned long long m = sh < 62u ? ((t.m << left) + ((1ull << sh) >> 1)) >> sh : 0ull;
    return t.neg ? -(long long)m : (long long)m;
}
__device__ __forceinline__ double fx_value(long long t, unsigned emax, int left) {
    if (t == 0) return 0.0;
    const int k = (int)emax - 1075 - left;
    const long long d = __double_as_longlong(__ll2double_rn(t));
    const int ed = (int)(d >> 52 & 0x7ff) + k;
    if (ed <= 0 || ed >= 0x7ff) return ldexp(__longlong_as_double(d), k);
    return __longlong_as_double(d + ((long long)k << 52));
}
constexpr int fx_log2(int n) { return n <= 1 ? 0 : 1 + fx_log2((n + 1) / 2); }

// sum of N values of this lane
template <int N>
__device__ __forceinline__ double fx_sum(const double (&v)[N]) {
    constexpr int kLeft = 10 - fx_log2(N);
    FxTerm t[N];
    unsigned emax = 1;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        t[k] = fx_term(v[k]);
        emax = max(emax, t[k].e);
    }
    if (emax >= 0x7ffu) {  // infinities and NaN
        double s = v[0];
#pragma unroll
        for (int k = 1; k < N; ++k) s += v[k];
        return s;
    }
    long long s = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) s += fx_align(t[k], emax, kLeft);
    return fx_value(s, emax, kLeft);
}

// sum over all lanes and N values per lane, in every lane
template <int N>
__device__ __forceinline__ double warp_fx_sum(const double (&v)[N]) {
    constexpr int kLeft = 5 - fx_log2(N);
    FxTerm t[N];
    unsigned emax = 1;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        t[k] = fx_term(v[k]);
        emax = max(emax, t[k].e);
    }
    emax = __reduce_max_sync(0xffffffffu, emax);
    if (emax >= 0x7ffu) {
        double s = v[0];
#pragma unroll
        for (int k = 1; k < N; ++k) s += v[k];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        return s;
    }
    long long s = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) s += fx_align(t[k], emax, kLeft);
    // three limbs of 24, 24 and 16 bits, each summed over the warp
    const int l0 = (int)(s & 0xffffff), l1 = (int)(s >> 24 & 0xffffff), l2 = (int)(s >> 48);
    const long long tot = (long long)__reduce_add_sync(0xffffffffu, l0) +
                          ((long long)__reduce_add_sync(0xffffffffu, l1) << 24) +
                          ((long long)__reduce_add_sync(0xffffffffu, l2) << 48);
    return fx_value(tot, emax, kLeft);
}

// Eight sums over the warp at once (a transposing butterfly): round 16 swaps
// half of the values between the half-warps, round 8 and 4 likewise, then two
// plain xor rounds; 9 shuffles instead of 40, in independent chains.  Lane l
// returns the total of value warp_sum8_index(l); the tree is fixed, so the
// result does not depend on timing.
__device__ __forceinline__ int warp_sum8_index(int lane) {
    return ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
}
template <class T>
__device__ __forceinline__ T warp_sum8(const T (&v)[8], int lane) {
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    T a4[4], a2[2];
#pragma unroll
    for (int q = 0; q < 4; ++q)
        a4[q] = (b4 ? v[q + 4] : v[q]) + __shfl_xor_sync(0xffffffffu, b4 ? v[q] : v[q + 4], 16);
#pragma unroll
    for (int q = 0; q < 2; ++q)
        a2[q] = (b3 ? a4[q + 2] : a4[q]) + __shfl_xor_sync(0xffffffffu, b3 ? a4[q] : a4[q + 2], 8);
    T a1 = (b2 ? a2[1] : a2[0]) + __shfl_xor_sync(0xffffffffu, b2 ? a2[0] : a2[1], 4);
    a1 += __shfl_xor_sync(0xffffffffu, a1, 2);
    a1 += __shfl_xor_sync(0xffffffffu, a1, 1);
    return a1;
}

// the same for doubles in fixed point
__device__ __forceinline__ double warp_fx_sum8(const double (&v)[8], int lane) {
    constexpr int kLeft = 5;
    FxTerm t[8];
    unsigned em[8], all = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        t[k] = fx_term(v[k]);
        em[k] = __reduce_max_sync(0xffffffffu, t[k].e);
        all = max(all, em[k]);
    }
    if (all >= 0x7ffu) return warp_sum8(v, lane);
    long long s[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) s[k] = fx_align(t[k], em[k], kLeft);
    const long long tot = warp_sum8(s, lane);
    const int idx = warp_sum8_index(lane);
    unsigned e = em[0];
#pragma unroll
    for (int k = 1; k < 8; ++k) e = idx == k ? em[k] : e;
    return fx_value(tot, e, kLeft);
}

// The stopping test sqrt(rr) / normb <= tol on squares (a square root and a division are 1,200 cycles of the FP64 pipe):
// rr <= the threshold.  A negative tol holds for no rr.  NaN where the square of tol normb leaves the doubles' normal
// range; the test then takes the roots.
__device__ __forceinline__ double rr_threshold(double tol, double normb) {
    const double t = tol * normb;
    if (tol < 0.) return -1.;
    return tol == 0. || (t > 1e-150 && t < 1e150) ? t * t : __longlong_as_double(0x7fffffffffffffffll);
}
static __device__ __noinline__ bool rr_reached_roots(double rr, double tol, double normb) { return sqrt(rr) / normb <= tol; }
__device__ __forceinline__ bool rr_reached(double rr, double thr, double tol, double normb) {
    // NaN told by its bits: an FP64 comparison more is 64 cycles on the path of every iteration
    if (((unsigned)__double2hiint(thr) >> 19 & 0xfffu) == 0xfffu) return rr_reached_roots(rr, tol, normb);
    return rr <= thr;
}
// x / rho and rho / x with the reciprocal of rho formed beforehand, off the path of the reduction that gives x; by division
// where that reciprocal could overflow or underflow
__device__ __forceinline__ bool rho_plain(double rho) {
    return ((unsigned)__double2hiint(rho) >> 20 & 0x7ffu) - 32u < 1984u;  // 2^-991 <= |rho| < 2^993
}
static __device__ __noinline__ double rho_quotient(double x, double y) { return x / y; }
__device__ __forceinline__ double by_rho(double x, double rho, double rho_inv) {
    return rho_plain(rho) ? x * rho_inv : rho_quotient(x, rho);
}
__device__ __forceinline__ double rho_by(double rho, double rho_inv, double x) {
    return rho_plain(rho) ? 1.0 / (x * rho_inv) : rho_quotient(rho, x);
}

template <int NV, class T>
__device__ void block_partials(T (&v)[NV], double* part /* [nblocks][NV] */) {
    __shared__ double red[NV][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int k = 0; k < NV; ++k) {
        const T x = warp_sum(v[k]);
        if (lane == 0) red[k][w] = (double)x;
    }
    __syncthreads();
    if (w == 0)
        for (int k = 0; k < NV; ++k) {
            double x = lane < nw ? red[k][lane] : 0.;
            x = warp_sum(x);
            if (lane == 0) part[(size_t)blockIdx.x * NV + k] = x;
        }
    __syncthreads();
}

// Scalar state of a persistent Krylov solve in global memory.  Only thread 0
// of the block that completes a grid step (the last to arrive) writes it, and
// only between its reduction and the barrier release; every block copies it
// into shared memory after the release.  FP64 arithmetic issues at a small
// fraction of the FP32 rate on GB300, so the scalar recurrences (divisions,
// square roots, convergence tests) run once per step instead of once per
// thread.  8-byte fields, copied as words.
struct KryScal {
    double rho, r_last, normb, resid, alpha, beta;
    long long it, done, converged, true_res, updates, pad;
};
constexpr int kScalWords = (int)(sizeof(KryScal) / 8);

// grid_sync_reduce with a scalar update: the last block sums the partials in a
// fixed order and thread 0 runs f(sums, state) on the global state.
template <int NV, class F>
__device__ bool grid_step(const GridSync& g, const double* part, KryScal* gsc, KryScal& ssc, F f) {
    __shared__ int last;
    __shared__ double red[NV][32];
    __shared__ int st;
    __syncthreads();
    unsigned my = 0;
    if (threadIdx.x == 0) {
        volatile unsigned* vgen = g.gen;
        my = *vgen;
        __threadfence();
        last = atomicAdd(g.count, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last) {
        __threadfence();
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
        for (int k = 0; k < NV; ++k) {
            double x = 0.;
            for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) x += __ldcg(part + (size_t)b * NV + k);
            x = warp_sum(x);
            if (lane == 0) red[k][w] = x;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double sums[NV];
            for (int k = 0; k < NV; ++k) {
                double x = 0.;
                for (int ww = 0; ww < nw; ++ww) x += red[k][ww];
                sums[k] = x;
            }
            f(sums, *gsc);
            __threadfence();
            *g.count = 0;
            __threadfence();
            atomicAdd(g.gen, 1u);
        }
    } else if (threadIdx.x == 0) {
        volatile unsigned* vgen = g.gen;
        long long spins = 0;
        while (*vgen == my) {
            if (++spins > kSpinLimit) {
                atomicCAS(g.status, 0, TF_ERR_WATCHDOG);
                break;
            }
            if (spins > 256) __nanosleep(32);
        }
        __threadfence();
    }
    if (threadIdx.x == 0) {
        st = *((volatile int*)g.status);
        const unsigned long long* src = reinterpret_cast<const unsigned long long*>(gsc);
        unsigned long long* dst = reinterpret_cast<unsigned long long*>(&ssc);
        for (int k = 0; k < kScalWords; ++k) dst[k] = __ldcg(src + k);
    }
    __syncthreads();
    return st == 0;
}

// ---------------------------------------------------------------------------
// barrier + all-reduce on one monotone arrival counter
//
// Every block publishes NV partial sums, arrives on a 64-bit counter that is
// never reset inside a launch and waits until the counter reaches
// (epoch + 1) * gridDim.x.  Arrival is a release of the whole block's writes:
// bar.sync, then thread 0's fence (cumulative over the writes the barrier
// ordered before it), then the atomic; the wait ends with an acquire (the
// polling load and a fence) before the block's bar.sync.  Then
// every block sums all partials itself, warp k taking value k over the blocks
// in one fixed order, so all blocks hold bitwise the same sums and derive the
// same scalars: the critical path is the arrival, one poll round trip and one
// load of the partials, with no last-arriver reduction and no published
// result to read back.  Partials alternate between two buffers by epoch
// parity; a block cannot be more than one barrier ahead of a reader.
// ---------------------------------------------------------------------------
constexpr int kArMax = 8;  // values per all-reduce (<= warps per block)

struct GridAR {
    unsigned long long* count;  // arrivals since launch (zeroed by the host)
    float* partf;               // [2][nblocks][kArMax]
    double* partd;              // [2][nblocks][kArMax]
    int* status;
};

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_release_add_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void fence_acquire_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Arrive and wait for all blocks of this epoch; false after a watchdog
// timeout.  Arrival is one release reduction by thread 0 after the block's
// bar.sync (cumulative: it releases every write the barrier ordered before
// it); the wait spins on relaxed loads and ends with one acquire fence, which
// the closing bar.sync extends to the whole block.  No sequentially
// consistent fence is needed on either side.
__device__ __forceinline__ bool ar_arrive_wait(const GridAR& g, unsigned long long epoch, int* st_sh) {
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned long long target = (epoch + 1) * (unsigned long long)gridDim.x;
        red_release_add_u64(g.count, 1ull);
        long long spins = 0;
        while (ld_relaxed_u64(g.count) < target) {
            if (++spins > kSpinLimit) {
                atomicCAS(g.status, 0, TF_ERR_WATCHDOG);
                break;
            }
            if (spins > 256) __nanosleep(32);
        }
        fence_acquire_gpu();
        *st_sh = *((volatile int*)g.status);
    }
    __syncthreads();
    return *st_sh == 0;
}

template <class T>
__device__ __forceinline__ T* ar_part(const GridAR& g);
template <>
__device__ __forceinline__ float* ar_part<float>(const GridAR& g) { return g.partf; }
template <>
__device__ __forceinline__ double* ar_part<double>(const GridAR& g) { return g.partd; }

// the kArMax values of one block's record (L2 only: written by other SMs)
__device__ __forceinline__ void ar_load_record(const float* p, float (&r)[8]) {
    const float4 a = __ldcg(reinterpret_cast<const float4*>(p)), b = __ldcg(reinterpret_cast<const float4*>(p) + 1);
    r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w;
    r[4] = b.x; r[5] = b.y; r[6] = b.z; r[7] = b.w;
}
__device__ __forceinline__ void ar_load_record(const double* p, double (&r)[8]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const double2 a = __ldcg(reinterpret_cast<const double2*>(p) + q);
        r[2 * q] = a.x;
        r[2 * q + 1] = a.y;
    }
}
static_assert(kArMax == 8, "records of eight values");

// Sums v[k] over every thread of the grid into out[k] (identical in all
// threads).  Call from all threads of every block, in uniform control flow.
// FP64 values: fixed-point warp sums, value k in warp k, so no chain of FP64
// adds is left on the way.
template <int NV>
__device__ bool grid_allreduce_f64(const GridAR& g, unsigned long long& epoch, const double (&v)[NV],
                                   double (&out)[NV]) {
    static_assert(NV >= 1 && NV <= kArMax, "all-reduce width");
    __shared__ double red[NV][32];
    __shared__ double res[NV];
    __shared__ int st;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double* part = g.partd + (size_t)(epoch & 1) * gridDim.x * kArMax;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const double one[1] = {v[k]};
        const double tot = warp_fx_sum(one);
        if (lane == 0) red[k][w] = tot;
    }
    __syncthreads();
    for (int k = w; k < NV; k += nw) {
        const double one[1] = {lane < nw ? red[k][lane] : 0.};
        const double x = warp_fx_sum(one);
        if (lane == 0) part[(size_t)blockIdx.x * kArMax + k] = x;
    }
    if (!ar_arrive_wait(g, epoch, &st)) return false;
    ++epoch;
    for (int k = w; k < NV; k += nw) {
        double x = 0.;
        for (unsigned c0 = 0; c0 < gridDim.x; c0 += 256) {
            double p[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const unsigned b = c0 + 32 * u + lane;
                p[u] = b < gridDim.x ? __ldcg(part + (size_t)b * kArMax + k) : 0.;
            }
            const double s = warp_fx_sum(p);
            x = c0 ? x + s : s;
        }
        if (lane == 0) res[k] = x;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; ++k) out[k] = res[k];
    return true;
}

// the same sums in T = float (or double, above)
template <class T, int NV>
__device__ bool grid_allreduce(const GridAR& g, unsigned long long& epoch, const T (&v)[NV], T (&out)[NV]) {
    static_assert(NV >= 1 && NV <= kArMax, "all-reduce width");
    if constexpr (sizeof(T) == 8) {
        return grid_allreduce_f64<NV>(g, epoch, v, out);
    } else {
        constexpr int kReadWarps = 8;  // warps that load block records
        __shared__ T red[kArMax][32];
        __shared__ T tot_w[kArMax][kReadWarps];
        __shared__ T res[kArMax];
        __shared__ int st;
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
        T* part = ar_part<T>(g) + (size_t)(epoch & 1) * gridDim.x * kArMax;
        // all NV sums of a warp at once (transposing butterfly, 9 shuffles)
        const int idx = warp_sum8_index(lane);
        {
            T v8[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v8[k] = k < NV ? v[k] : T(0);
            const T tot = warp_sum8(v8, lane);
            if ((lane & 3) == 0 && idx < NV) red[idx][w] = tot;
        }
        __syncthreads();
        if (threadIdx.x < NV) {
            T x = T(0);
            for (int ww = 0; ww < nw; ++ww) x += red[threadIdx.x][ww];
            part[(size_t)blockIdx.x * kArMax + threadIdx.x] = x;
        }
        if (!ar_arrive_wait(g, epoch, &st)) return false;
        ++epoch;
        // the block records (kArMax values: 32 or 64 bytes, 16-byte loads, one
        // L2 sector request per record) are spread over up to kReadWarps warps,
        // one record per lane, so that they are in flight at once; each warp sums
        // its records (in the order of the chunks it took, then the fixed shuffle
        // tree), and NV lanes of warp 0 add the warp totals in warp order, so
        // every block derives the same bits.
        const int nchunks = (int)((gridDim.x + 31) / 32);
        const int nread = nw < kReadWarps ? nw : kReadWarps;
        if (w < nread) {
            T acc[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[k] = T(0);
            for (int ch = w; ch < nchunks; ch += nread) {
                const unsigned b = (unsigned)ch * 32u + (unsigned)lane;
                if (b < gridDim.x) {
                    T rec[8];
                    ar_load_record(part + (size_t)b * kArMax, rec);
#pragma unroll
                    for (int k = 0; k < NV; ++k) acc[k] += rec[k];
                }
            }
            const T tot = warp_sum8(acc, lane);
            if ((lane & 3) == 0 && idx < NV) tot_w[idx][w] = tot;
        }
        __syncthreads();
        if (threadIdx.x < NV) {
            const int nused = nchunks < nread ? nchunks : nread;
            T x = tot_w[threadIdx.x][0];
            for (int ww = 1; ww < nused; ++ww) x += tot_w[threadIdx.x][ww];
            res[threadIdx.x] = x;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < NV; ++k) out[k] = res[k];
        return true;
    }
}

// ---------------------------------------------------------------------------
// All-reduce in one trip: packed fixed-point accumulators
//
// grid_allreduce makes three dependent trips to L2 (the release of the
// partials, the poll of the arrival counter, the read of the partials).  Here
// a block adds its partial sum as an integer to one 64-bit word per value,
// together with its arrival: bits 0..7 count the arrivals, bits 8..15 the
// arrivals whose partial did not fit, bits 16..63 hold the sum.  A block that
// polls the word sees the finished sum with the last arrival: one atomic add
// and one poll.  Integer sums do not depend on the order of arrival, so every
// block gets the same bits.  The unit of a value follows from its previous sum,
// which all blocks know: an FP32 value takes one word with 2^38 units to that
// sum, an FP64 value two (a 48-bit high and a 40-bit low part) with 2^76.  The
// blocks repeat the reduction with grid_allreduce when a block's sum exceeds twice
// (8 times in FP64; on fewer than 128 blocks more) the previous sum or is not
// finite, and when the sum is smaller than 2^-6 of it.  So the rounding of all the terms
// that are aligned to the unit - the blocks' sums in FP32, at most 255; the
// threads' values in FP64, at most 2^17 - adds up to at most 255 x 2^-39 x 2^6 =
// 2^-25 (2^17 x 2^-77 x 2^6 = 2^-54) of the sum: half of what rounding it to its
// type costs.  (Without the last condition a GMRES basis vector a thousand times
// shorter than the one before lost its norm, and the solver stagnated.)
//
// Words are never reset: two buffers alternate, and a block remembers the value
// each of its words had when it last read it (a block is at most one reduction
// ahead of a reader).  Grids of up to 255 blocks.
//
// Measured on GB300, 152 blocks of 512 threads, per reduction of 6 words: 2.70
// (grid_allreduce of 6 FP32 values) -> 0.93 us, 1.26 us with the fence that
// publishes other data; grid_allreduce of 2 FP64 values takes 3.63 us.
// ---------------------------------------------------------------------------
constexpr int kPkWords = 256;  // words of one buffer
constexpr int kPkMaxBlocks = 255;
constexpr int kPkUnknown = -100000;  // no previous sum: grid_allreduce

struct PackedAR {
    unsigned long long* w;  // [2][kPkWords], zeroed before the launch
    int* status;
};

__device__ __forceinline__ void red_relaxed_add_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
constexpr int kPkUnits32 = 38, kPkUnits64 = 76;  // log2 of the units to the previous sum
constexpr int kPkDrop32 = 6, kPkDrop64 = 6;      // exponents a sum may fall below the previous one
// log2 of the range of a block's sum in a word of 48 bits
__device__ __forceinline__ int pk_range() { return 15 + __clz((int)gridDim.x); }
__device__ __forceinline__ unsigned long long pk_word(long long t, bool bad) {
    return bad ? 257ull : ((unsigned long long)t << 16) + 1ull;
}
// waits for all blocks on word p; *diff = what they added since `last`
__device__ __forceinline__ bool pk_wait(const unsigned long long* p, unsigned long long& last, int* status,
                                        unsigned long long* diff) {
    long long spins = 0;
    unsigned long long v;
    while ((((v = ld_relaxed_u64(p)) - last) & 255ull) != gridDim.x) {
        if (++spins > kSpinLimit) {
            atomicCAS(status, 0, TF_ERR_WATCHDOG);
            return false;
        }
        if (spins > 256) __nanosleep(32);
    }
    *diff = v - last;
    last = v;
    return true;
}
__device__ __forceinline__ bool pk_misfit(unsigned long long diff) { return (diff >> 8 & 255ull) != 0; }
__device__ __forceinline__ long long pk_sum(unsigned long long diff) { return (long long)diff >> 16; }

// exponent of a sum (2^e <= |x| < 2^(e+1)); kPkUnknown for zero and non-finite values
__device__ __forceinline__ int pk_exp(float x) {
    const int e = __float_as_int(x) >> 23 & 0xff;
    return e == 0 || e == 255 ? kPkUnknown : e - 127;
}
__device__ __forceinline__ int pk_exp(double x) {
    const int e = __double2hiint(x) >> 20 & 0x7ff;
    return e == 0 || e == 2047 ? kPkUnknown : e - 1023;
}
// x in units of 2^(E - kPkUnits64) as hi 2^40 + lo (both with the sign of x); *bad when it exceeds 2^87 units
__device__ __forceinline__ void pk_fix(double x, int E, long long* hi, long long* lo, bool* bad) {
    const long long b = __double_as_longlong(x);
    const int e = (int)(b >> 52) & 0x7ff;
    const unsigned long long m = ((unsigned long long)b & 0xfffffffffffffull) | (e ? 1ull << 52 : 0ull);
    const int s = max(e, 1) - 1075 - E + kPkUnits64;
    *bad = e == 2047 || s > 34;
    const unsigned __int128 t = s >= 0 ? (unsigned __int128)m << min(s, 34)
                                       : (unsigned __int128)(s > -62 ? (m + ((1ull << -s) >> 1)) >> -s : 0ull);
    const long long h = (long long)(t >> 40), l = (long long)(t & 0xffffffffffull);
    *hi = b < 0 ? -h : h;
    *lo = b < 0 ? -l : l;
}
// the same value with 0 <= lo < 2^40; false when it does not fit a partial's range
__device__ __forceinline__ bool pk_carry(long long* hi, long long* lo) {
    *hi += *lo >> 40;
    *lo &= 0xffffffffffll;
    const long long cap = 1ll << pk_range();
    return *hi < cap && *hi > -cap;
}
// x in units of 2^(E - kPkUnits32), rounded to nearest; *bad when it exceeds a block's range
__device__ __forceinline__ long long pk_fix(float x, int E, bool* bad) {
    const int b = __float_as_int(x), e = b >> 23 & 0xff;
    const long long m = (b & 0x7fffff) | (e ? 0x800000 : 0);
    const int s = max(e, 1) - 150 - E + kPkUnits32, top = pk_range() - 24;  // m 2^(e - 150)
    *bad = e == 255 || s > top;
    const long long t = s >= 0 ? m << min(s, top) : (s > -40 ? (m + ((1ll << -s) >> 1)) >> -s : 0ll);
    return b < 0 ? -t : t;
}
__device__ __forceinline__ float pk_value(long long t, int E) { return ldexpf(__ll2float_rn(t), E - kPkUnits32); }

// hi 2^40 + lo as a 62-bit magnitude and a shift
__device__ __forceinline__ unsigned long long pk_magnitude(long long hi, long long lo, bool* neg, int* shift) {
    const __int128 t = ((__int128)hi << 40) + lo;
    *neg = t < 0;
    unsigned __int128 u = *neg ? (unsigned __int128)(-t) : (unsigned __int128)t;
    *shift = 0;
    const unsigned long long top = (unsigned long long)(u >> 62);  // |t| < 2^96
    if (top) {
        *shift = 64 - __clzll((long long)top);
        u >>= *shift;
    }
    return (unsigned long long)u;
}
__device__ __forceinline__ double pk_value(long long hi, long long lo, int E) {
    bool neg;
    int k;
    const unsigned long long u = pk_magnitude(hi, lo, &neg, &k);
    const double d = fx_value((long long)u, (unsigned)(E - kPkUnits64 + k + 1075 + 4096), 4096);
    return neg ? -d : d;
}

// per-thread state of the packed reductions of one set of values
struct PkState {
    unsigned long long last[2] = {0ull, 0ull};
    int E = kPkUnknown;  // lane k (FP32), lanes 2 k and 2 k + 1 (FP64): exponent of value k's last sum
    unsigned epoch = 0;
    bool known = false;  // uniform over the grid
};
// one word of a reduction: adds, waits; 0: *diff holds what the blocks added, 1: to be repeated, 2: watchdog
__device__ __forceinline__ int pk_exchange(const PackedAR& g, unsigned epoch, unsigned long long (&last)[2], int word,
                                           long long t, bool fits, unsigned long long* diff) {
    unsigned long long* p = g.w + (epoch & 1) * kPkWords + word;
    red_relaxed_add_u64(p, pk_word(t, !fits));
    if (!pk_wait(p, epoch & 1 ? last[1] : last[0], g.status, diff)) return 2;
    return pk_misfit(*diff) ? 1 : 0;
}

// Sums of NV <= 8 values over the grid, as grid_allreduce.  publish: the
// blocks' earlier writes are visible to every block afterwards.
template <int NV>
__device__ bool packed_allreduce(const PackedAR& g, PkState& pk, const GridAR& slow, unsigned long long& slow_epoch,
                                 const float (&v)[NV], float (&out)[NV], bool publish) {
    static_assert(NV <= 8, "two words per value");
    __shared__ float red[NV][32];
    __shared__ float res[NV];
    __shared__ int state;  // 0: done, 1: repeat, 2: watchdog
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (pk.known) {
        {
            float v8[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v8[k] = k < NV ? v[k] : 0.f;
            const float tot = warp_sum8(v8, lane);
            const int idx = warp_sum8_index(lane);
            if ((lane & 3) == 0 && idx < NV) red[idx][w] = tot;
        }
        __syncthreads();
        if (w == 0) {
            int st = 0;
            float x = 0.f;
            if (lane < NV)
                for (int ww = 0; ww < nw; ++ww) x += red[lane][ww];
            if (publish) __threadfence();
            if (lane < NV) {
                bool bad;
                const long long t = pk_fix(x, pk.E, &bad);
                unsigned long long diff = 0;
                st = pk_exchange(g, pk.epoch, pk.last, lane, t, !bad, &diff);
                x = pk_value(pk_sum(diff), pk.E);
                res[lane] = x;
                const int e = pk_exp(x);
                if (e < pk.E - kPkDrop32) st = max(st, 1);
                pk.E = e;
            }
            if (publish) fence_acquire_gpu();
            st = (int)__reduce_max_sync(0xffffffffu, (unsigned)st);
            if (lane == 0) state = st;
        }
        ++pk.epoch;
        __syncthreads();
        if (state == 2) return false;
        if (state == 0) {
#pragma unroll
            for (int k = 0; k < NV; ++k) out[k] = res[k];
            return true;
        }
    }
    if (!grid_allreduce<float, NV>(slow, slow_epoch, v, out)) return false;
    bool ok = true;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int e = pk_exp(out[k]);
        ok &= e != kPkUnknown;
        if (lane == k) pk.E = e;
    }
    pk.known = ok;
    return true;
}

template <int NV>
__device__ bool packed_allreduce(const PackedAR& g, PkState& pk, const GridAR& slow, unsigned long long& slow_epoch,
                                 const double (&v)[NV], double (&out)[NV], bool publish) {
    static_assert(NV <= 8, "two words per value");
    __shared__ long long redh[NV][32], redl[NV][32];
    __shared__ double res[NV];
    __shared__ int sE[NV];
    __shared__ int redb[32];
    __shared__ int state;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (pk.known) {
        // every thread's values in the common units, summed over the warp in limbs of 20 bits
        bool bad = false;
        auto warp_add = [](long long x, bool three) -> long long {
            const int a = (int)(x & 0xfffff), b = three ? (int)(x >> 20 & 0xfffff) : (int)(x >> 20);
            long long r = (long long)__reduce_add_sync(0xffffffffu, a) + ((long long)__reduce_add_sync(0xffffffffu, b) << 20);
            if (three) r += (long long)__reduce_add_sync(0xffffffffu, (int)(x >> 40)) << 40;
            return r;
        };
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            long long h, l;
            bool bk;
            pk_fix(v[k], __shfl_sync(0xffffffffu, pk.E, 2 * k), &h, &l, &bk);
            bad |= bk;
            h = warp_add(h, true);
            l = warp_add(l, false);
            if (lane == 0) {
                redh[k][w] = h;
                redl[k][w] = l;
            }
        }
        bad = __any_sync(0xffffffffu, bad);
        if (lane == 0) redb[w] = bad;
        __syncthreads();
        if (w == 0) {
            long long t = 0;
            bool fits = !__any_sync(0xffffffffu, lane < nw && redb[lane]);
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                // the warps' sums: |h| < 2^53, |l| < 2^46
                long long h = lane < nw ? redh[k][lane] : 0ll, l = lane < nw ? redl[k][lane] : 0ll;
                h = warp_add(h, true);
                l = warp_add(l & 0xffffffffffll, false) + (warp_add(l >> 40, false) << 40);
                const bool f = pk_carry(&h, &l);
                if (lane >> 1 == k) {
                    t = lane & 1 ? l : h;
                    fits &= f;
                }
            }
            int st = 0;
            if (publish) __threadfence();
            long long s = 0;
            if (lane < 2 * NV) {
                unsigned long long diff = 0;
                st = pk_exchange(g, pk.epoch, pk.last, lane, t, fits, &diff);
                s = lane & 1 ? (long long)(diff >> 16) : pk_sum(diff);  // low parts are not negative
            }
            const long long lo = __shfl_down_sync(0xffffffffu, s, 1);
            if (lane < 2 * NV && !(lane & 1)) {
                const double x = pk_value(s, lo, pk.E);
                const int e = pk_exp(x);
                if (e < pk.E - kPkDrop64) st = max(st, 1);
                pk.E = e;
                res[lane >> 1] = x;
                sE[lane >> 1] = e;
            }
            if (publish) fence_acquire_gpu();
            st = (int)__reduce_max_sync(0xffffffffu, (unsigned)st);
            if (lane == 0) state = st;
        }
        ++pk.epoch;
        __syncthreads();
        if (state == 2) return false;
        if (state == 0) {
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                out[k] = res[k];
                if (lane >> 1 == k) pk.E = sE[k];
            }
            return true;
        }
    }
    if (!grid_allreduce<double, NV>(slow, slow_epoch, v, out)) return false;
    bool ok = true;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int e = pk_exp(out[k]);
        ok &= e != kPkUnknown;
        if (lane >> 1 == k) pk.E = e;
    }
    pk.known = ok;
    return true;
}

// plain barrier on the same counter
__device__ __forceinline__ bool grid_sync_ar(const GridAR& g, unsigned long long& epoch) {
    __shared__ int st;
    if (!ar_arrive_wait(g, epoch, &st)) return false;
    ++epoch;
    return true;
}

// Shared-memory copy of a contiguous run of SELL slots: slots [base, base +
// cap) of the column and value arrays, laid out as in global memory.  A slice
// whose slots all lie in the run is read from shared memory.
template <class T>
struct SellCache {
    const int32_t* col = nullptr;  // shared memory
    const T* val = nullptr;
    int32_t base = 0, cap = 0;
};

// n columns of a slot row from cp / vp (already at slot lane of the first
// column, 32 slots per column): in blocks of eight, the loads of the next
// block issued while the gathers of the current block are in flight, so a
// lane keeps up to 16 independent loads outstanding and n columns cost
// ceil(n/8) gather latencies.  SH: cp / vp point to shared memory.  Loads past
// n are masked and the multiply-adds past n are skipped (n is warp-uniform,
// so no FP64 pipe time goes to padding).  Terms are summed in CSR order.
template <bool SH, class T, class XL>
__device__ __forceinline__ T sell_row_walk(const int32_t* __restrict__ cp, const T* __restrict__ vp, int32_t n,
                                           XL xload) {
    constexpr int U = 8;
    auto ldc = [](const int32_t* p) { return SH ? *p : __ldg(p); };
    auto ldv = [](const T* p) { return SH ? *p : __ldg(p); };
    T acc = T(0);
    int32_t cn[U];
    T vn[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const bool in = u < n;
        cn[u] = in ? ldc(cp + 32 * u) : -1;
        vn[u] = in ? ldv(vp + 32 * u) : T(0);
    }
    for (int32_t k = 0; k < n; k += U) {
        T xv[U], vv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            xv[u] = cn[u] >= 0 ? xload(cn[u]) : T(0);
            vv[u] = vn[u];
        }
        const int32_t kn = k + U;
        if (kn < n) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const bool in = kn + u < n;
                cn[u] = in ? ldc(cp + 32 * (kn + u)) : -1;
                vn[u] = in ? ldv(vp + 32 * (kn + u)) : T(0);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (k + u < n) acc += vv[u] * xv[u];
    }
    return acc;
}

// Slot row of a SELL matrix times the vector given by xload(col), over the
// slice columns [c0, c0 + n), accumulated in T; from the shared-memory copy
// when the cache holds the whole slice.
template <class T, class XL>
__device__ __forceinline__ T sell_row_range(const int32_t* __restrict__ ptr, const int32_t* __restrict__ col,
                                            const T* __restrict__ val, int64_t s, int lane, int32_t c0, int32_t n,
                                            XL xload, const SellCache<T>& cache = SellCache<T>()) {
    const int32_t ps = __ldg(ptr + s), p0 = ps + 32 * c0;
    if (cache.cap > 0 && ps >= cache.base && __ldg(ptr + s + 1) - cache.base <= cache.cap)
        return sell_row_walk<true, T>(cache.col + (p0 - cache.base) + lane, cache.val + (p0 - cache.base) + lane, n,
                                      xload);
    return sell_row_walk<false, T>(col + p0 + lane, val + p0 + lane, n, xload);
}

// the whole slot row (all columns of slice s)
template <class T, class XL>
__device__ __forceinline__ T sell_row(const int32_t* __restrict__ ptr, const int32_t* __restrict__ col,
                                      const T* __restrict__ val, int64_t s, int lane, XL xload) {
    const int32_t w = (__ldg(ptr + s + 1) - __ldg(ptr + s)) >> 5;
    return sell_row_range<T>(ptr, col, val, s, lane, 0, w, xload);
}

// ---------------------------------------------------------------------------
// Balanced SELL product of one block.  The block takes the slices [s0, s1)
// (at most kBalMaxSlices) and splits their total column count T evenly over
// its NW warps: warp j walks the column positions [jT/NW, (j+1)T/NW) of the
// concatenated slices, so a wide slice is shared by several warps and every
// warp walks about T/NW columns (the gather chain of the slowest warp no
// longer follows the widest slice).  A slice that lies wholly inside one warp's
// range is emitted by that warp; a split slice's partial sums go to shared
// memory and the warp holding its last column adds them in column order
// (deterministic).  emit(slice, value) is called by all 32 lanes of a warp;
// zero-width slices (empty rows) are emitted too.  All threads of the block
// must call this, in uniform control flow; it ends with a block barrier, so
// what emit wrote to shared memory can be read right after.
// ---------------------------------------------------------------------------
constexpr int kBalMaxSlices = 64;

// First slice of part b of nparts when the slices [0, nslices) are split at
// equal work, work(s) = columns(s) + kBalRowCost per slice (the per-row
// updates that follow the product), using the SELL offsets ptr (32 x columns,
// a prefix sum): the largest s with work before s <= b W / nparts.
constexpr int kBalRowCost = 4;
__device__ __forceinline__ int64_t balanced_part_start(const int32_t* __restrict__ ptr, int64_t nslices, int64_t b,
                                                       int64_t nparts) {
    if (b <= 0) return 0;
    if (b >= nparts) return nslices;
    const int64_t total = (int64_t)(__ldg(ptr + nslices) >> 5) + kBalRowCost * nslices;
    const int64_t target = total * b / nparts;
    int64_t lo = 0, hi = nslices;  // work(lo) <= target < work(hi + 1)
    while (lo < hi) {
        const int64_t mid = (lo + hi + 1) >> 1;
        if ((int64_t)(__ldg(ptr + mid) >> 5) + kBalRowCost * mid <= target) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

template <int NW, class T, int MAXS = kBalMaxSlices>
struct BalShared {
    int32_t P[MAXS + 1];
    T tail[NW][32];
};

// A warp's part of the planned columns: slices [lo, hi) of which the first began
// in warp ja when ja >= 0.
struct WalkRange {
    int32_t g0, g1;  // columns
    int lo, hi, ja;
};

// The column prefix of the slices [s0, s0 + S) into sh.P (one block
// barrier); a block that walks the same slices repeatedly plans once.
template <int NW, class T>
__device__ __forceinline__ void sell_block_plan(BalShared<NW, T>& sh, const int32_t* __restrict__ ptr, int64_t s0,
                                                int S) {
    const int lane = threadIdx.x & 31, j = threadIdx.x >> 5;
    if (j == 0) {
        int carry = 0;
        for (int b = 0; b < S; b += 32) {
            const int i = b + lane;
            int w = i < S ? (__ldg(ptr + s0 + i + 1) - __ldg(ptr + s0 + i)) >> 5 : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += t;
            }
            if (i < S) sh.P[i + 1] = carry + w;
            carry += __shfl_sync(0xffffffffu, w, 31);
        }
        if (lane == 0) sh.P[0] = 0;
    }
    __syncthreads();
}

// The part of this thread's warp: binary searches, 0.2 to 0.5 us of shared memory
// latency, so a block that walks the same slices repeatedly keeps it (in shared
// memory: a register array of it spills in the resident solvers).
template <int NW, class T, int MAXS>
__device__ __forceinline__ WalkRange sell_block_range(const BalShared<NW, T, MAXS>& sh, int S) {
    const int j = threadIdx.x >> 5;
    const int32_t Tot = sh.P[S];
    WalkRange r;
    r.g0 = (int32_t)((int64_t)j * Tot / NW);
    r.g1 = (int32_t)((int64_t)(j + 1) * Tot / NW);
    // first slice that overlaps [g0, ..) or starts at g0 (zero width included)
    int lo = 0, hi = S;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (sh.P[mid + 1] > r.g0 || sh.P[mid] >= r.g0) hi = mid;
        else lo = mid + 1;
    }
    r.lo = lo;
    // first slice beyond: it starts at g1 or later (the last warp takes the empty slices at the end)
    hi = S;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (!(sh.P[mid] < r.g1 || (j == NW - 1 && sh.P[mid] == Tot))) hi = mid;
        else lo = mid + 1;
    }
    r.hi = lo;
    r.ja = -1;
    if (r.lo < r.hi && sh.P[r.lo] < r.g0) {
        int ja = j - 1;
        while (ja > 0 && (int32_t)((int64_t)ja * Tot / NW) > sh.P[r.lo]) --ja;
        r.ja = ja;
    }
    return r;
}

// The product over planned slices (sh.P holds the prefix of [s0, s0 + S)):
// row(slice, c0, n) returns one lane's partial sum over the slice columns
// [c0, c0 + n); T needs T(0) and +.
template <int NW, class T, int MAXS, class ROW, class EMIT>
__device__ __forceinline__ void sell_block_walk_range(BalShared<NW, T, MAXS>& sh, int64_t s0, int S, const WalkRange& wr,
                                                      ROW row, EMIT emit) {
    const int lane = threadIdx.x & 31, j = threadIdx.x >> 5;
    const int32_t g0 = wr.g0, g1 = wr.g1;
    const int lo = wr.lo, hi = wr.hi;
    T head = T(0);
    bool end = false;  // the first slice began in another warp and ends here
    if (lo < hi) {
        int32_t pa = sh.P[lo];
        for (int i = lo; i < hi; ++i) {
            const int32_t pb = sh.P[i + 1];
            const int32_t c0 = g0 > pa ? g0 - pa : 0;
            const int32_t c1 = (g1 < pb ? g1 : pb) - pa;
            const T acc = row(s0 + i, c0, c1 > c0 ? c1 - c0 : 0);
            const bool starts = pa >= g0, ends = pb <= g1;
            if (starts && ends) {
                emit(s0 + i, acc);
            } else if (ends) {
                head = acc;
                end = true;
            } else {
                sh.tail[j][lane] = acc;
            }
            pa = pb;
        }
    }
    __syncthreads();
    if (end) {
        // warps from the one holding the slice's first column up to this one
        const int32_t Tot = sh.P[S];
        T sum = T(0);
        for (int jj = wr.ja; jj < j; ++jj) {
            const int32_t a0 = (int32_t)((int64_t)jj * Tot / NW), a1 = (int32_t)((int64_t)(jj + 1) * Tot / NW);
            if (a1 > a0) sum = sum + sh.tail[jj][lane];
        }
        emit(s0 + lo, sum + head);
    }
    __syncthreads();  // emits visible to the block; sh.tail free for the next call
}

// The same for a single walk: without the searches for the end of the range.
template <int NW, class T, int MAXS, class ROW, class EMIT>
__device__ __forceinline__ void sell_block_walk_fn(BalShared<NW, T, MAXS>& sh, int64_t s0, int S, ROW row, EMIT emit) {
    const int lane = threadIdx.x & 31, j = threadIdx.x >> 5;
    const int32_t Tot = sh.P[S];
    const int32_t g0 = (int32_t)((int64_t)j * Tot / NW), g1 = (int32_t)((int64_t)(j + 1) * Tot / NW);
    // first slice that overlaps [g0, ..) or starts at g0 (zero width included)
    int lo = 0, hi = S;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (sh.P[mid + 1] > g0 || sh.P[mid] >= g0) hi = mid;
        else lo = mid + 1;
    }
    T head = T(0);
    int hslice = -1;
    for (int i = lo; i < S; ++i) {
        const int32_t pa = sh.P[i], pb = sh.P[i + 1];
        if (!(pa < g1 || (j == NW - 1 && pa == Tot))) break;
        const int32_t c0 = g0 > pa ? g0 - pa : 0;
        const int32_t c1 = (g1 < pb ? g1 : pb) - pa;
        const T acc = row(s0 + i, c0, c1 > c0 ? c1 - c0 : 0);
        const bool starts = pa >= g0, ends = pb <= g1;
        if (starts && ends) {
            emit(s0 + i, acc);
        } else if (ends) {
            head = acc;
            hslice = i;
        } else {
            sh.tail[j][lane] = acc;
        }
    }
    __syncthreads();
    if (hslice >= 0) {
        // warps from the one holding the slice's first column up to this one
        const int32_t pa = sh.P[hslice];
        int ja = j - 1;
        while (ja > 0 && (int32_t)((int64_t)ja * Tot / NW) > pa) --ja;
        T sum = T(0);
        for (int jj = ja; jj < j; ++jj) {
            const int32_t a0 = (int32_t)((int64_t)jj * Tot / NW), a1 = (int32_t)((int64_t)(jj + 1) * Tot / NW);
            if (a1 > a0) sum = sum + sh.tail[jj][lane];
        }
        emit(s0 + hslice, sum + head);
    }
    __syncthreads();  // emits visible to the block; sh.tail free for the next call
}

template <int NW, class T, class XL, class EMIT>
__device__ __forceinline__ void sell_block_walk(BalShared<NW, T>& sh, const int32_t* __restrict__ ptr,
                                                const int32_t* __restrict__ col, const T* __restrict__ val,
                                                int64_t s0, int S, XL xload, EMIT emit,
                                                const SellCache<T>& cache = SellCache<T>()) {
    const int lane = threadIdx.x & 31;
    sell_block_walk_fn(
        sh, s0, S,
        [&](int64_t s, int32_t c0, int32_t n) { return sell_row_range<T>(ptr, col, val, s, lane, c0, n, xload, cache); },
        emit);
}

template <int NW, class T, class XL, class EMIT>
__device__ __forceinline__ void sell_block_balanced(BalShared<NW, T>& sh, const int32_t* __restrict__ ptr,
                                                    const int32_t* __restrict__ col, const T* __restrict__ val,
                                                    int64_t s0, int S, XL xload, EMIT emit,
                                                    const SellCache<T>& cache = SellCache<T>()) {
    sell_block_plan<NW, T>(sh, ptr, s0, S);
    sell_block_walk<NW, T>(sh, ptr, col, val, s0, S, xload, emit, cache);
}

// n columns of one slot row: translated columns cp[32 k] (shared memory),
// values vp[32 k] (shared memory when VSH, else global: a pointer to either makes
// every load generic), vector xs (shared memory).  Terms are summed in column order.
template <bool VSH, class T>
__device__ __forceinline__ T res_row(const uint16_t* __restrict__ cp, const T* __restrict__ vp, int32_t n,
                                     const T* __restrict__ xs) {
    constexpr int U = 8;
    T acc = T(0);
    for (int32_t k = 0; k < n; k += U) {
        T xv[U], vv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (k + u < n) {
                vv[u] = VSH ? vp[32 * (k + u)] : __ldg(vp + 32 * (k + u));
                xv[u] = xs[cp[32 * (k + u)]];
            } else {
                vv[u] = T(0);
                xv[u] = T(0);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (k + u < n) acc += vv[u] * xv[u];
    }
    return acc;
}

#define TF_SLICE_LOOP(nslices, s)                                                    \
    const int64_t warp__ = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;   \
    const int64_t nwarp__ = ((int64_t)gridDim.x * blockDim.x) >> 5;                  \
    for (int64_t s = warp__; s < (nslices); s += nwarp__)

// Slice order of the persistent kernels, where every warp walks several
// slices between two grid barriers and the barrier waits for the slowest
// warp.  The SELL rows are sorted by length inside windows of
// kSellWinSlices slices (512 rows), so slice rank k of every window has about
// the same width and rank 0 is the widest: taking slices in storage order
// hands the widest slice of every window to the same warp index.  Here
// position p runs rank-major (p = k * nwin + win, slice win * 16 + k: widest
// ranks first), and warp w of n takes positions w, 2n-1-w, 2n+w, ...: the
// passes alternate direction, so each warp pairs wide slices with narrow ones.
// A bijection on [0, nslices) for nslices a multiple of kSellWinSlices;
// warp-uniform control flow.
constexpr int kSellWinSlices = 16;
__device__ __forceinline__ int64_t slice_at_rank(int64_t pos, int64_t nwin) {
    return (pos % nwin) * kSellWinSlices + pos / nwin;
}
#define TF_SLICE_LOOP_BAL(nslices, s)                                                                     \
    const int64_t bw__ = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;                          \
    const int64_t bn__ = ((int64_t)gridDim.x * blockDim.x) >> 5;                                          \
    const int64_t bwin__ = (nslices) / kSellWinSlices;                                                    \
    for (int64_t bi__ = 0; bi__ * bn__ < (nslices); ++bi__)                                               \
        for (int64_t bp__ = bi__ * bn__ + ((bi__ & 1) ? bn__ - 1 - bw__ : bw__),                          \
                     s = bp__ < (nslices) ? slice_at_rank(bp__, bwin__) : -1;                             \
             s >= 0; s = -1)

}  // namespace tf

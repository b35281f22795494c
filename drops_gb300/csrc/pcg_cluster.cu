// Jacobi-PCG of one system per CTA or thread-block cluster (num/krylovsolver.h:
// 107-189): the batched solver and small single systems.
//
// A cluster of C CTAs (1 to 8) solves a system; its rows are split into C
// contiguous ranges.  A CTA sorts its rows by length, so that its slices of 32
// rows carry little padding, and writes its share of the matrix column-major
// with 16-bit columns (cluster slots): 6 bytes per entry, read coalesced, where
// CSR rows on a few lanes took 8 bytes in up to 9 sectors per request.  The whole
// vector p (every CTA advances p = z + beta p itself), and r, q and 1/d of the CTA's
// rows lie in shared memory; x and as many slices of the matrix as fit follow, the
// rest of them lie in global memory (L2).  The column work is split evenly over the
// warps.  A reduction is one block reduction; with C > 1 also one 8-byte store to
// every CTA of the cluster (distributed shared memory) and a hardware cluster
// barrier, and z goes through L2 (written by its owner, read whole by the others).
//
// V = float: the mixed solver (FP32 iterations, the iterate x in FP64, the FP64
// residual b - A x in place of the FP32 one whenever that has dropped by
// rel_update or claims convergence); V = double: the reference's recurrences.
//
// What bounds it (256 ellipsoids of 16^3 to 64^3 cubes, mixed, C = 2, us per iteration):
// the product 5.1, of which the gathers from p (3.5 bank conflicts of 32 random words)
// take about 3.4; the second reduction 3.0 with the FP64 update of x under its wait (an
// FP64 instruction holds the pipe 64 cycles); the first 1.6; the FP64 residuals 1.7 (every
// 20th iteration); p and r 0.9.  k_batch_pcg took 34.6 at 8,180 rows where this takes
// 25.6, 15.0, 9.4, 7.1 on 1, 2, 4, 8 CTAs; the whole batch took 33.7 ms and takes 13.0.
// 1,024 threads (64 registers, spills to an L1 of a few KB) took 15.6 ms, two CTAs of
// 256 threads per SM 16.3.  FP64 is bound by the FP64 pipe of its SMs: 8,180 rows 102 ->
// 27.9, 18.2, 13.7 on 2, 4, 8 CTAs.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "krylov_dev.cuh"

namespace tf {

namespace {

template <class V>
constexpr int kClThreads = 512;  // 128 registers a thread
constexpr int kClMaxCtas = 8;
constexpr int kClMaxSlices = 1024;            // 32,768 rows per CTA
constexpr int kClMaxRows = 32 * kClMaxSlices;
constexpr int kClMaxSlots = 65536;            // 16-bit columns

struct ClArgs {
    int count;               // systems
    const int32_t* order;    // queue order (nullptr: 0, 1, ...)
    const int64_t* rows;     // count + 1 row starts of all systems (nullptr: one system of m rows)
    int64_t m;
    const int32_t* rowptr;
    const int32_t* col;
    const double* val;
    const double* b;
    double* x;
    unsigned char* scratch;  // per CTA: cl_scratch bytes, for what the shared memory does not hold
    size_t scratch_cta;
    void* z;                 // [cluster][pcap] values of V in slot order (C > 1)
    int32_t* slotmap;        // [m] cluster slot of every row
    int* queue;
    int* out_iter;           // per system: iterations k, or -1-k when not converged
    double* out_resid;       // per system: reached residual
    int* out_updates;        // FP64 residuals of the last system (may be nullptr)
    int max_iter, rel;
    double tol, rel_update;
    int pcap, ncap;          // slots of the largest system and of the largest share
    int ecap;                // entries of a CTA's scratch
    int room;                // bytes of dynamic shared memory
};

struct ClShared {
    int next, done, converged, refine;
    double rho, rho_inv, alpha, beta, thr_tol, thr_last, normb, rr;
    unsigned char* scratch;  // this CTA's
    void* z;                 // this cluster's
    double slot[2][3][kClMaxCtas];  // partial sums of the cluster's CTAs, two buffers
    double part[3][32];
};

__device__ __forceinline__ unsigned cl_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cl_size() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cl_id() {
    unsigned r;
    asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
    return r;
}
// barrier over all threads of the cluster; writes before the arrival (shared,
// distributed shared and global memory) are visible to the cluster after the wait.
// .aligned: a warp's lanes execute it together, so they meet before it.
__device__ __forceinline__ void cl_arrive() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cl_wait() {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cl_sync() {
    cl_arrive();
    cl_wait();
}
__device__ __forceinline__ uint32_t cl_map(const void* p, unsigned rank) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void cl_store(const double* p, unsigned rank, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(cl_map(p, rank)), "d"(v) : "memory");
}
__device__ __forceinline__ void cl_store(const int* p, unsigned rank, int v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cl_map(p, rank)), "r"(v) : "memory");
}
__device__ __forceinline__ double cl_widen(float x) { return widen_f32(x); }
__device__ __forceinline__ double cl_widen(double x) { return x; }

__host__ __device__ inline size_t cl_up(size_t b) { return (b + 127) & ~(size_t)127; }
template <class V>
__host__ __device__ inline size_t cl_fixed(int P, int NS) {  // shared memory: row numbers, slice places, p
    return cl_up((size_t)NS * 4) + cl_up((size_t)NS / 32 * 4) + cl_up((size_t)P * sizeof(V));
}
template <class V>
size_t cl_scratch(int ncap, int ecap) {
    return cl_up((size_t)ncap * 8) + cl_up((size_t)ecap * sizeof(V)) + cl_up((size_t)ecap * 2);
}

// n columns of one slot row: columns cp[32 k], values vp[32 k] (loads of the next
// eight issued while the current eight are multiplied), vector xs in shared memory
template <class V>
__device__ __forceinline__ V cl_row(const uint16_t* cp, const V* vp, int32_t n, const V* xs) {
    constexpr int U = sizeof(V) == 4 ? 8 : 4;
    V acc = V(0);
    int cn[U];
    V vn[U];
    auto load = [&](int32_t k) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool in = k + u < n;
            cn[u] = in ? cp[32 * (k + u)] : 0;
            vn[u] = in ? vp[32 * (k + u)] : V(0);
        }
    };
    load(0);
    for (int32_t k = 0; k < n; k += U) {
        V xv[U], vv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            xv[u] = k + u < n ? xs[cn[u]] : V(0);
            vv[u] = vn[u];
        }
        if (k + U < n) load(k + U);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (k + u < n) acc += vv[u] * xv[u];
    }
    return acc;
}

template <class V>
struct ClTriple {
    V a, b, c;
};
template <class V>
struct ClStep {
    double x;
    V p;
};
// f(t, load(t)) for this thread's t < n, U loads at a time (a store between two loads of possibly
// aliasing arrays would serialise them)
template <int U, class LOAD, class F>
__device__ __forceinline__ void cl_each(int n, LOAD load, F f) {
    const int nt = blockDim.x;
    for (int t0 = threadIdx.x; t0 < n; t0 += U * nt) {
        decltype(load(0)) w[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (t0 + u * nt < n) w[u] = load(t0 + u * nt);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (t0 + u * nt < n) f(t0 + u * nt, w[u]);
    }
}

template <class V>
__global__ void __launch_bounds__(kClThreads<V>, 1) k_pcg_cluster(ClArgs a) {
    constexpr bool kMixed = sizeof(V) == 4;
    constexpr int NT = kClThreads<V>, NW = NT / 32, kEach = 2;
    extern __shared__ __align__(128) unsigned char cl_dyn[];
    __shared__ ClShared sh;
    __shared__ BalShared<NW, V, kClMaxSlices> bsh;
    __shared__ WalkRange wrs[NW];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int C = (int)cl_size(), rank = (int)cl_rank();
    // pointers that are used once per phase wait in shared memory (registers)
    if (threadIdx.x == 0) {
        sh.scratch = a.scratch + (size_t)blockIdx.x * a.scratch_cta;
        sh.z = reinterpret_cast<V*>(a.z) + (size_t)cl_id() * a.pcap;
    }
    int flip = 0;

    // Sums of NV values over the cluster; f runs on thread 0 of every CTA with the sums (the same bits in every
    // CTA: partials in CTA order, added in fixed point), `meanwhile` on every thread while it waits for the others.
    // Ends with a block barrier.
    auto cluster_sum = [&](auto tag, const auto& v, auto meanwhile, auto f) {
        constexpr int NV = decltype(tag)::value;
        using T = std::decay_t<decltype(v[0])>;
        flip ^= 1;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            double s;
            if constexpr (sizeof(T) == 4) {
                s = cl_widen(warp_sum(v[k]));
            } else {
                const double one[1] = {v[k]};
                s = warp_fx_sum(one);
            }
            if (lane == 0) sh.part[k][warp] = s;
        }
        __syncthreads();
        if (C == 1) {
            if (warp == 0) {
                double o[NV];
#pragma unroll
                for (int k = 0; k < NV; ++k) {
                    const double one[1] = {lane < NW ? sh.part[k][lane] : 0.};
                    o[k] = warp_fx_sum(one);
                }
                if (lane == 0) f(o);
            }
            meanwhile();
            __syncthreads();
            return;
        }
        if (warp < NV) {
            const double one[1] = {lane < NW ? sh.part[warp][lane] : 0.};
            const double s = warp_fx_sum(one);
            if (lane < C) cl_store(&sh.slot[flip][warp][rank], (unsigned)lane, s);
        }
        cl_arrive();
        meanwhile();
        cl_wait();
        if (warp == 0) {
            double o[NV];
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                const double one[1] = {lane < C ? sh.slot[flip][k][lane] : 0.};
                o[k] = warp_fx_sum(one);
            }
            if (lane == 0) f(o);
        }
        __syncthreads();
    };
    using N1 = std::integral_constant<int, 1>;
    using N2 = std::integral_constant<int, 2>;
    using N3 = std::integral_constant<int, 3>;

    cl_sync();  // every CTA of the cluster has started: its shared memory may be written
    for (;;) {
        if (rank == 0 && threadIdx.x == 0) {
            const int k = atomicAdd(a.queue, 1);
            for (int c = 0; c < C; ++c) cl_store(&sh.next, (unsigned)c, k);
        }
        cl_sync();
        const int qk = sh.next;
        if (qk >= a.count) return;
        const int inst = a.order ? a.order[qk] : qk;
        const int64_t r0 = a.rows ? a.rows[inst] : 0, r1 = a.rows ? a.rows[inst + 1] : a.m;
        const int nrows = (int)(r1 - r0);
        const int per = ((nrows + 32 * C - 1) / (32 * C)) * 32;  // rows of a CTA's share
        const int own0 = min(rank * per, nrows), n = min(per, nrows - own0);
        const int S = (n + 31) / 32, NS = S * 32, P = per * C;
        // shared memory: row numbers, p, r, 1/d, q, then x, then as much of the matrix as fits
        size_t used = cl_fixed<V>(P, NS);
        int32_t* const srow = reinterpret_cast<int32_t*>(cl_dyn);
        int32_t* const soff = reinterpret_cast<int32_t*>(cl_dyn + cl_up((size_t)NS * 4));  // entry in shared memory, or -1
        V* const p = reinterpret_cast<V*>(cl_dyn + cl_up((size_t)NS * 4) + cl_up((size_t)S * 4));
        V* const own = p + rank * per;
        const size_t nb = cl_up((size_t)NS * sizeof(V)), xb = cl_up((size_t)NS * 8);
        V* const rs = reinterpret_cast<V*>(cl_dyn + used);
        V* const ds = reinterpret_cast<V*>(cl_dyn + used + nb);
        V* const qs = reinterpret_cast<V*>(cl_dyn + used + 2 * nb);
        used += 3 * nb;
        const bool x_sh = used + xb <= (size_t)a.room;
        double* const xs = reinterpret_cast<double*>(x_sh ? cl_dyn + used : sh.scratch);
        if (x_sh) used += xb;
        const int sme = (int)((a.room - used) / (sizeof(V) + 2) & ~(size_t)63);  // entries in shared memory
        V* const sval = reinterpret_cast<V*>(cl_dyn + used);
        uint16_t* const scol = reinterpret_cast<uint16_t*>(sval + sme);
        auto gval = [&] { return reinterpret_cast<V*>(sh.scratch + cl_up((size_t)a.ncap * 8)); };
        auto gcol = [&] { return reinterpret_cast<uint16_t*>(gval() + a.ecap); };

        // ---- rows of the share by descending length (ties by row): bitonic sort of (length, row) ----
        {
            uint32_t* const kk = reinterpret_cast<uint32_t*>(srow);
            // keys beyond n would need a power of two of room; missing partners count as the largest key
            int np = 32;
            while (np < n) np <<= 1;
            for (int t = threadIdx.x; t < n; t += NT) {
                const int64_t row = r0 + own0 + t;
                const int len = min(a.rowptr[row + 1] - a.rowptr[row], 0xffff);
                kk[t] = (uint32_t)(0xffff - len) << 16 | (uint32_t)t;
            }
            __syncthreads();
            // ascending sort of any length: the first step of every merge mirrors, so absent keys stay at the end
            for (int size = 2; size <= np; size <<= 1) {
                for (int stride = size >> 1; stride > 0; stride >>= 1) {
                    for (int i = threadIdx.x; i < np / 2; i += NT) {
                        int x, y;
                        if (stride == size >> 1) {
                            const int g = i / stride, o = i % stride;
                            x = g * size + o;
                            y = g * size + size - 1 - o;
                        } else {
                            x = 2 * stride * (i / stride) + i % stride;
                            y = x + stride;
                        }
                        if (y < n) {
                            const uint32_t u = kk[x], v = kk[y];
                            if (u > v) {
                                kk[x] = v;
                                kk[y] = u;
                            }
                        }
                    }
                    __syncthreads();
                }
            }
            for (int t = threadIdx.x; t < NS; t += NT) {
                const int row = t < n ? own0 + (int)(kk[t] & 0xffffu) : -1;
                srow[t] = row;
                if (t < n) a.slotmap[r0 + row] = rank * per + t;
            }
            __syncthreads();
            // the first row of a slice is its longest; the column prefix of the slices
            if (warp == 0) {
                int carry = 0;
                for (int s0 = 0; s0 < S; s0 += 32) {
                    const int s = s0 + lane;
                    int inc = 0;
                    if (s < S) {
                        const int64_t row = r0 + srow[32 * s];
                        inc = a.rowptr[row + 1] - a.rowptr[row];
                    }
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y = __shfl_up_sync(0xffffffffu, inc, o);
                        if (lane >= o) inc += y;
                    }
                    if (s < S) bsh.P[s + 1] = carry + inc;
                    carry += __shfl_sync(0xffffffffu, inc, 31);
                }
                if (lane == 0) bsh.P[0] = 0;
            }
        }
        cl_sync();  // slot numbers of the whole system written
        // slices that fit the scratch; what is left (a share above the host's estimate) is read from the CSR
        int fit = S;
        if (32 * bsh.P[S] > a.ecap) {
            int lo = 0, hi = S;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (32 * bsh.P[mid] <= a.ecap) lo = mid;
                else hi = mid - 1;
            }
            fit = lo;
        }
        // the slices kept in shared memory are spread evenly, so every warp's part is as much in L2 as the others'
        if (threadIdx.x == 0) {
            const int64_t tot = bsh.P[S], cap = sme / 32;
            int acc = 0;
            for (int s = 0; s < S; ++s) {
                const int e = bsh.P[s + 1], w = e - bsh.P[s];
                const bool in = cap >= tot || (acc + w <= cap && (acc + w) * tot <= cap * e);
                soff[s] = in ? 32 * acc : -1;
                if (in) acc += w;
            }
        }
        __syncthreads();
        if (lane == 0) wrs[warp] = sell_block_range(bsh, fit);
        __syncwarp();
        for (int s = warp; s < S; s += NW) {
            const int row = srow[32 * s + lane];
            int32_t k0 = 0, k1 = 0;
            double di = 0.;
            if (row >= 0) {
                k0 = a.rowptr[r0 + row];
                k1 = a.rowptr[r0 + row + 1];
            }
            const int w = bsh.P[s + 1] - bsh.P[s], t = 32 * s + lane, so = soff[s];
#pragma unroll 4
            for (int k = 0; k < w; ++k) {
                V v = V(0);
                int c = rank * per + t;
                if (k0 + k < k1) {
                    const int32_t j = __ldg(a.col + k0 + k);
                    const double av = __ldg(a.val + k0 + k);
                    v = (V)av;
                    c = __ldcg(a.slotmap + j);
                    if (j == r0 + row) di = av;  // the Jacobi diagonal (SolveGSstep<PB_JAC0> scans the row for it)
                }
                if (s < fit) {
                    if (so >= 0) {
                        sval[so + 32 * k + lane] = v;
                        scol[so + 32 * k + lane] = (uint16_t)c;
                    } else {
                        gval()[32 * (bsh.P[s] + k) + lane] = v;
                        gcol()[32 * (bsh.P[s] + k) + lane] = (uint16_t)c;
                    }
                }
            }
            ds[t] = row >= 0 ? (V)(1.0 / (kMixed ? (double)(V)di : di)) : V(0);
            xs[t] = row >= 0 ? a.x[r0 + row] : 0.;
        }
        for (int t = threadIdx.x; t < P; t += NT) p[t] = V(0);
        __syncthreads();

        // q = A p on the share; returns this thread's part of <q, p>
        auto product = [&]() -> V {
            V pq = V(0);
            sell_block_walk_range(
                bsh, 0, fit, wrs[warp],
                [&](int64_t s, int32_t c0, int32_t nn) {
                    const int so = soff[s];
                    if (so >= 0) {
                        const int e = so + 32 * c0 + lane;
                        return res_row<true, V>(scol + e, sval + e, nn, p);
                    }
                    const int e = 32 * (bsh.P[s] + c0) + lane;
                    return cl_row<V>(gcol() + e, gval() + e, nn, p);
                },
                [&](int64_t s, V v) {
                    const int t = 32 * (int)s + lane;
                    qs[t] = v;
                    pq += v * own[t];
                });
            for (int s = fit + warp; s < S; s += NW) {  // beyond the room: from the CSR arrays
                const int t = 32 * s + lane, row = srow[t];
                V v = V(0);
                if (row >= 0)
                    for (int32_t k = a.rowptr[r0 + row]; k < a.rowptr[r0 + row + 1]; ++k)
                        v += (V)__ldg(a.val + k) * p[__ldcg(a.slotmap + __ldg(a.col + k))];
                qs[t] = v;
                pq += v * own[t];
            }
            if (fit < S) __syncthreads();
            return pq;
        };
        // r = b - A x in FP64 from the CSR arrays, four lanes to a row, z = r / d
        int updates = 0;
        auto true_residual = [&](bool first) {
            double v[3] = {0., 0., 0.};
            const int sub = lane & 3;
            // Row starts, entries and x are dependent trips to L2: those of the next rows are in flight meanwhile.  A warp
            // takes 8 rows at a time; four times 8 rows are summed by one exchange, after which every lane holds one
            // row (an FP64 instruction holds the pipe 64 cycles however few lanes are active).
            constexpr int U = 4;
            auto slot = [&](int i) { return 32 * (warp + NW * (i >> 2)) + 8 * (i & 3) + (lane >> 2); };
            auto starts = [&](int i, int32_t& k, int32_t& k1) {
                const int t = slot(i), row = t < NS ? srow[t] : -1;
                k = k1 = 0;
                if (row >= 0) {
                    k = __ldg(a.rowptr + r0 + row) + sub;
                    k1 = __ldg(a.rowptr + r0 + row + 1);
                }
            };
            auto entries = [&](int32_t k, int32_t k1, int32_t (&j)[U], double (&av)[U]) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const bool in = k + 4 * u < k1;
                    j[u] = in ? __ldg(a.col + k + 4 * u) : (int32_t)r0;
                    av[u] = in ? __ldg(a.val + k + 4 * u) : 0.;
                }
            };
            int32_t k, k1, kn, kn1, j[U];
            double av[U], part[4];
            starts(0, k, k1);
            starts(1, kn, kn1);
            entries(k, k1, j, av);
            for (int s = warp; s < S; s += NW) {
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const int i = 4 * ((s - warp) / NW) + h;
                    double xv[U], ax = 0.;
#pragma unroll
                    for (int u = 0; u < U; ++u) xv[u] = __ldcg(a.x + j[u]);
                    int32_t jn[U], kp, kp1;
                    double an[U];
                    entries(kn, kn1, jn, an);
                    starts(i + 2, kp, kp1);
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (k + 4 * u < k1) ax += av[u] * xv[u];
                    for (k += 4 * U; k < k1; k += 4) ax += __ldg(a.val + k) * __ldcg(a.x + __ldg(a.col + k));
                    part[h] = ax;
                    k = kn;
                    k1 = kn1;
                    kn = kp;
                    kn1 = kp1;
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        j[u] = jn[u];
                        av[u] = an[u];
                    }
                }
                __syncwarp();
                // lane 4 g + h gets the sum of rows 8 h + g: over sub, halving the rows held
                const bool b0 = sub & 1, b1 = sub & 2;
                const double e0 = __shfl_xor_sync(0xffffffffu, b0 ? part[0] : part[1], 1);
                const double e1 = __shfl_xor_sync(0xffffffffu, b0 ? part[2] : part[3], 1);
                const double f0 = (b0 ? part[1] : part[0]) + e0, f1 = (b0 ? part[3] : part[2]) + e1;
                const double ax = (b1 ? f1 : f0) + __shfl_xor_sync(0xffffffffu, b1 ? f0 : f1, 2);
                const int t = 32 * s + 8 * sub + (lane >> 2), row = srow[t];
                V zi = V(0), ri = V(0);
                if (row >= 0) {
                    const double bi = a.b[r0 + row], r = bi - ax;
                    ri = (V)r;
                    zi = ri * ds[t];
                    v[0] += r * r;
                    if (first) v[1] += bi * bi;
                    v[2] += (double)zi * (double)ri;
                }
                rs[t] = ri;
                if (C > 1) ((V*)sh.z)[rank * per + t] = zi;
            }
            ++updates;
            cluster_sum(N3{}, v, [] {}, [&](const double* o) {
                if (first) {
                    double nb = sqrt(o[1]);
                    if (nb == 0.0 || !a.rel) nb = 1.0;
                    sh.normb = nb;
                    sh.thr_tol = rr_threshold(a.tol, nb);
                    sh.beta = 0.;
                } else {
                    sh.beta = by_rho(o[2], sh.rho, sh.rho_inv);
                }
                sh.rr = o[0];
                sh.thr_last = kMixed ? a.rel_update * a.rel_update * o[0] : 0.;
                sh.rho = o[2];
                sh.converged = rr_reached(o[0], sh.thr_tol, a.tol, sh.normb);
            });
        };
        int it = 0;
        bool refine = true;
        for (;;) {
            if (refine) {
                if (it > 0) {
                    for (int t = threadIdx.x; t < NS; t += NT)
                        if (srow[t] >= 0) a.x[r0 + srow[t]] = xs[t];
                    if (C == 1) __syncthreads();
                    else cl_sync();
                }
                true_residual(it == 0);
                if (sh.converged || it >= a.max_iter) break;
            }
            // p = z + beta p: with C = 1 from the CTA's own r, else the whole vector from L2
            {
                const V beta = (V)sh.beta;
                // under the product: the divisor of the next alpha and beta
                if (threadIdx.x == 32) sh.rho_inv = 1.0 / sh.rho;
                if (C == 1) {
                    cl_each<kEach>(NS, [&](int t) { return ClTriple<V>{rs[t], ds[t], p[t]}; },
                               [&](int t, const ClTriple<V>& w) { p[t] = w.a * w.b + beta * w.c; });
                } else if constexpr (kMixed) {
                    float4* const p4 = reinterpret_cast<float4*>(p);
                    const float4* const z4 = reinterpret_cast<const float4*>(sh.z);
                    for (int t = threadIdx.x; t < P / 4; t += NT) {
                        const float4 zz = __ldcg(z4 + t);
                        float4 q = p4[t];
                        q.x = fmaf(beta, q.x, zz.x);
                        q.y = fmaf(beta, q.y, zz.y);
                        q.z = fmaf(beta, q.z, zz.z);
                        q.w = fmaf(beta, q.w, zz.w);
                        p4[t] = q;
                    }
                } else {
                    const V* const z = (const V*)sh.z;
                    for (int t = threadIdx.x; t < P; t += NT) p[t] = __ldcg(z + t) + beta * p[t];
                }
            }
            __syncthreads();
            ++it;
            {
                const V v[1] = {product()};
                cluster_sum(N1{}, v, [] {}, [&](const double* o) { sh.alpha = rho_by(sh.rho, sh.rho_inv, o[0]); });
            }
            {
                const double alpha = sh.alpha;
                const V al = (V)alpha;
                V v[2] = {V(0), V(0)};
                V* const z = (V*)sh.z + rank * per;
                cl_each<kEach>(NS, [&](int t) { return ClTriple<V>{rs[t], qs[t], ds[t]}; },
                           [&](int t, const ClTriple<V>& w) {
                               const V r = w.a - al * w.b;
                               const V zi = r * w.c;
                               rs[t] = r;
                               if (C > 1) z[t] = zi;
                               v[0] += r * r;
                               v[1] += zi * r;
                           });
                // x += alpha p (FP64) under the wait
                auto update_x = [&] {
                    cl_each<kEach>(NS, [&](int t) { return ClStep<V>{xs[t], own[t]}; },
                               [&](int t, const ClStep<V>& w) { xs[t] = w.x + alpha * cl_widen(w.p); });
                };
                cluster_sum(N2{}, v, update_x, [&](const double* o) {
                    sh.rr = o[0];
                    if (kMixed) {
                        sh.refine = o[0] <= sh.thr_last || rr_reached(o[0], sh.thr_tol, a.tol, sh.normb) || it >= a.max_iter;
                        if (!sh.refine) {
                            sh.beta = by_rho(o[1], sh.rho, sh.rho_inv);
                            sh.rho = o[1];
                        }
                    } else {
                        sh.refine = 0;
                        sh.converged = rr_reached(o[0], sh.thr_tol, a.tol, sh.normb);
                        sh.done = sh.converged || it >= a.max_iter;
                        sh.beta = by_rho(o[1], sh.rho, sh.rho_inv);
                        sh.rho = o[1];
                    }
                });
            }
            refine = kMixed && sh.refine;
            if (!kMixed && sh.done) break;
        }
        if (!kMixed)
            for (int t = threadIdx.x; t < NS; t += NT)
                if (srow[t] >= 0) a.x[r0 + srow[t]] = xs[t];
        if (rank == 0 && threadIdx.x == 0) {
            a.out_iter[inst] = sh.converged ? it : -1 - it;
            a.out_resid[inst] = sqrt(sh.rr) / sh.normb;
            if (a.out_updates) *a.out_updates = updates;
        }
        cl_sync();  // the next system reuses the cluster's shared memory and z
    }
}

// Launch of `count` systems on clusters of C CTAs.  rows / nnz: of the largest system.
struct ClPlan {
    int C = 0, clusters = 0;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
};

// whether a system of `rows` rows fits a cluster of C CTAs
template <class V>
bool cl_fits(int64_t rows, int C, int64_t room) {
    const int64_t per = (rows + 32 * C - 1) / (32 * C) * 32;
    return per <= kClMaxRows && per * C <= kClMaxSlots && (int64_t)(cl_fixed<V>((int)(per * C), (int)per) + 3 * cl_up((size_t)per * sizeof(V))) <= room;
}

template <class V>
int cl_room(Context* c, int64_t* room) {
    TF_TRY(max_dynamic_smem(c, (const void*)k_pcg_cluster<V>, room));
    *room &= ~(int64_t)127;
    return TF_OK;
}

// fills plan, a.pcap .. a.room, a.scratch, a.z and a.slotmap (a.m given); *ok = false when the device has no room for it
template <class V>
int cl_plan(Context* c, int C, int count, int64_t rows, int64_t nnz, int64_t room, ClPlan* pl, ClArgs* a, bool* ok) {
    *ok = false;
    const void* fn = (const void*)k_pcg_cluster<V>;
    const int64_t per = (rows + 32 * C - 1) / (32 * C) * 32;
    a->ncap = (int)per;
    a->pcap = (int)(per * C);
    // sorted slices pad a share by at most 32 of its longest row; uneven shares take up to a quarter more
    const int64_t e = (C == 1 ? nnz : nnz / C + nnz / (4 * C)) + 32 * 128;
    if (e > (int64_t)1 << 28) return TF_OK;
    a->ecap = (int)((e + 63) & ~(int64_t)63);
    a->room = (int)room;
    pl->C = C;
    pl->attr.id = cudaLaunchAttributeClusterDimension;
    pl->attr.val.clusterDim.x = (unsigned)C;
    pl->attr.val.clusterDim.y = pl->attr.val.clusterDim.z = 1;
    pl->cfg = cudaLaunchConfig_t{};
    pl->cfg.blockDim = dim3(kClThreads<V>);
    pl->cfg.gridDim = dim3((unsigned)C);
    pl->cfg.dynamicSmemBytes = (size_t)room;
    pl->cfg.stream = c->stream;
    pl->cfg.attrs = &pl->attr;
    pl->cfg.numAttrs = 1;
    int n = 0;
    TF_CUDA(c, cudaOccupancyMaxActiveClusters(&n, fn, &pl->cfg));
    if (n < 1) return TF_OK;
    pl->clusters = std::min(n, count);
    pl->cfg.gridDim = dim3((unsigned)(pl->clusters * C));
    a->scratch_cta = cl_scratch<V>(a->ncap, a->ecap);
    TF_TRY(ensure_if_room(c, c->cl_scratch, a->scratch_cta * pl->clusters * C + c->cl_scratch_extra, ok));
    if (*ok) TF_TRY(ensure_if_room(c, c->cl_z, (size_t)a->pcap * pl->clusters, ok));
    if (*ok) TF_TRY(ensure_if_room(c, c->cl_slots, (size_t)a->m, ok));
    if (!*ok) {  // the other kernels need the memory that was had
        release(c->cl_scratch);
        release(c->cl_z);
        release(c->cl_slots);
        return TF_OK;
    }
    a->scratch = c->cl_scratch.p;
    a->z = c->cl_z.p;
    a->slotmap = c->cl_slots.p;
    return TF_OK;
}

template <class V>
int cl_launch(Context* c, const ClPlan& pl, ClArgs& a) {
    TF_CUDA(c, cudaMemsetAsync(a.queue, 0, sizeof(int), c->stream));
    void* args[] = {&a};
    cudaLaunchConfig_t cfg = pl.cfg;
    cudaLaunchAttribute attr = pl.attr;
    cfg.attrs = &attr;
    TF_CUDA(c, cudaLaunchKernelExC(&cfg, (const void*)k_pcg_cluster<V>, args));
    ++c->launches;
    return TF_OK;
}

}  // namespace

// CTAs of the cluster that solves a single system, 0 for the grid-wide kernels.
// The first solve on a pattern only: there the grid-wide kernels first build
// their layout (SELL windows, halo lists: about 250 us), which a cluster does
// not need; for later solves that layout pays, as it takes 5.4 (mixed) and 8.4
// (FP64) us an iteration.  First solve of the P1 sphere (whole pass, us; grid-wide
// / 8 CTAs / 1 CTA) at 2.8k non-zeros: FP64 899 / 740 / 697, mixed 910 / 741 / 664; at
// 5.8k: 1051 / 884 / 981, 1000 / 838 / 850; at 30k: 1940 / 1763, 1545 / 1454; at 49k:
// 2380 / 2687, 1781 / 1967; P2 at 36k: 1842 / 1770, 1490 / 1495.
int pcg_cluster_ctas(const Context* c, const CSR& A) {
    if (c->pcg_cluster >= 0) return c->pcg_cluster;
    if (c->pcg_shape_fixed || !c->pcg_resident || c->pcg_two_barrier) return 0;
    if (A.cluster_gen == A.pattern_gen || A.sell.pattern_gen == A.pattern_gen) return 0;
    return A.nnz <= 4096 ? 1 : A.nnz <= 32768 ? 8 : 0;
}

// One system on one cluster; *applied = false (nothing launched) when it does not fit.
template <class V>
int pcg_cluster(Context* c, CSR& A, int C, const double* b, double* x, int* max_iter, double* tol, int rel,
                bool* applied) {
    *applied = false;
    int64_t room = 0;
    TF_TRY(cl_room<V>(c, &room));
    if (A.m > INT32_MAX / 2 || !cl_fits<V>(A.m, C, room)) return TF_OK;
    ClPlan pl;
    ClArgs a{};
    a.m = A.m;
    TF_TRY(ensure(c, c->kry_iters, 4));
    TF_TRY(ensure(c, c->kry_resid, 1));
    TF_TRY(cl_plan<V>(c, C, 1, A.m, A.nnz, room, &pl, &a, applied));
    if (!*applied) return TF_OK;
    a.count = 1;
    a.rowptr = A.rowptr;
    a.col = A.colind;
    a.val = A.vals;
    a.b = b;
    a.x = x;
    a.queue = c->kry_iters.p;
    a.out_iter = c->kry_iters.p + 1;
    a.out_updates = c->kry_iters.p + 2;
    a.out_resid = c->kry_resid.p;
    a.max_iter = *max_iter;
    a.rel = rel;
    a.tol = *tol;
    a.rel_update = c->pcg_rel_update;
    TF_TRY(cl_launch<V>(c, pl, a));
    int* h = c->h_status + 8;  // pinned
    TF_CUDA(c, cudaMemcpyAsync(h, c->kry_iters.p + 1, 2 * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    TF_CUDA(c, cudaMemcpyAsync(h + 2, c->kry_resid.p, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    TF_CUDA(c, cudaStreamSynchronize(c->stream));
    A.cluster_gen = A.pattern_gen;
    c->last_refinements = h[1];
    *max_iter = h[0] >= 0 ? h[0] : -1 - h[0];
    std::memcpy(tol, h + 2, sizeof(double));
    return h[0] >= 0 ? TF_OK : set_err(c, TF_ERR_NOT_CONVERGED, "pcg: no convergence within max_iter");
}
template int pcg_cluster<float>(Context*, CSR&, int, const double*, double*, int*, double*, int, bool*);
template int pcg_cluster<double>(Context*, CSR&, int, const double*, double*, int*, double*, int, bool*);

// The batch (launch only, capturable once prepared): rows and nnz per instance on the host.
template <class V>
int batch_cluster_prepare(Context* c, CSR& A, BatchCluster* bc, bool* ok) {
    *ok = false;
    const int n = c->batch_count;
    int64_t room = 0, rmax = 0, nmax = 0;
    TF_TRY(cl_room<V>(c, &room));
    for (int i = 0; i < n; ++i) {
        rmax = std::max<int64_t>(rmax, c->h_batch_rows[i + 1] - c->h_batch_rows[i]);
        nmax = std::max(nmax, c->h_batch_nnz[i]);
    }
    if (rmax > INT32_MAX / 2) return TF_OK;
    // Estimated time on clusters of C CTAs: an iteration of n rows takes 5.3 us (two reductions, six phases) plus
    // 2.5 ns a row of the share beyond 700 (measured with 234 to 8,180 rows on 1, 2, 4, 8 CTAs: 5.9 / 7.2 / 7.1 / 7.1 us at
    // 234, 11.4 / 8.9 / 6.9 / 5.9 at 2,950, 25.6 / 15.0 / 9.4 / 7.1 at 8,180), the iterations grow with the square root of
    // the rows, and the launch ends with the longest system or with the queue.  Whole solves on 1, 2, 4, 8 CTAs
    // (ms): 256 ellipsoids of 16^3 to 64^3 cubes - / 13.1 / 16.8 / 30.9 (k_batch_pcg 33.0), 200 of 24^3 to 40^3
    // 21.1 / 20.1 / 23.0 / 31.2 (with assembly), 100 of 10^3 to 60^3 - / 22.0 / 17.4 / 21.0, 40 of 20^3 to 60^3
    // - / 16.1 / 11.8 / 10.6.  FP64: 6.3 us plus 5.3 ns a row of the share (the FP64 pipe) and 0.25 ns a row of the system
    // (p); solver alone in ms, k_batch_pcg and 1, 2, 4, 8 CTAs (-: does not fit): 256 of 16^3 to 64^3 91.1, - / - / - / 48.9;
    // 200 of 24^3 to 40^3 24.2, - / 8.4 / 12.2 / 22.2; 40 of 20^3 to 60^3 75.7, - / - / - / 7.9; 16 of 8^3 to 20^3 2.6,
    // 1.5 / 1.2 / 0.9 / 0.8.
    int C = 0;
    double best = 0.;
    for (int k = 1; k <= kClMaxCtas; k *= 2) {
        if (!cl_fits<V>(rmax, k, room)) continue;
        const double clusters = std::min(n, c->num_sms / k);
        double sum = 0., top = 0.;
        for (int i = 0; i < n; ++i) {
            const double rows = (double)(c->h_batch_rows[i + 1] - c->h_batch_rows[i]);
            const double us = sizeof(V) == 4 ? 5.3 + (k > 1 ? 1. : 0.) + 2.5e-3 * std::max(0., rows / k - 700.)
                                             : 6.3 + 5.3e-3 * rows / k + (k > 1 ? 0.25e-3 * rows : 0.);
            const double t = std::sqrt(rows) * us;
            sum += t;
            top = std::max(top, t);
        }
        const double est = std::max(top, sum / clusters);
        if (C == 0 || est < best) {
            C = k;
            best = est;
        }
    }
    if (c->pcg_cluster > 0) C = cl_fits<V>(rmax, c->pcg_cluster, room) ? c->pcg_cluster : 0;
    if (C == 0) return TF_OK;
    static_assert(sizeof(bc->blob) >= sizeof(ClPlan) + sizeof(ClArgs), "batch cluster blob");
    ClPlan pl;
    ClArgs a{};
    a.m = A.m;
    TF_TRY(cl_plan<V>(c, C, n, rmax, nmax, room, &pl, &a, ok));
    if (!*ok) return TF_OK;
    a.count = n;
    a.order = c->batch_order.p;
    a.rows = c->batch_rows.p;
    a.rowptr = A.rowptr;
    a.col = A.colind;
    a.val = A.vals;
    a.queue = c->batch_queue.p;
    a.out_iter = c->batch_iters.p;
    a.out_resid = c->batch_resid.p;
    std::memcpy(bc->blob, &pl, sizeof(pl));
    std::memcpy(bc->blob + sizeof(pl), &a, sizeof(a));
    bc->grid = (int)pl.cfg.gridDim.x;
    bc->mixed = sizeof(V) == 4;
    bc->ctas = C;
    bc->scratch = a.scratch;
    bc->z = a.z;
    return TF_OK;
}

int batch_cluster_launch(Context* c, const BatchCluster& bc, const double* b, double* x, int max_iter, double tol,
                         int rel) {
    ClPlan pl;
    ClArgs a;
    std::memcpy(&pl, bc.blob, sizeof(pl));
    std::memcpy(&a, bc.blob + sizeof(pl), sizeof(a));
    a.b = b;
    a.x = x;
    a.max_iter = max_iter;
    a.tol = tol;
    a.rel = rel;
    a.rel_update = c->batch_rel_update;
    return bc.mixed ? cl_launch<float>(c, pl, a) : cl_launch<double>(c, pl, a);
}
template int batch_cluster_prepare<float>(Context*, CSR&, BatchCluster*, bool*);
template int batch_cluster_prepare<double>(Context*, CSR&, BatchCluster*, bool*);

}  // namespace tf

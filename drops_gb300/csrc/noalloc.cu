// Jacobi-PCG for callers that cannot allocate device memory.
//
// tf_pcg_jacobi (krylov.cu) keeps its work vectors in memory owned by a
// tf_context, which allocates with cudaMalloc.  Some callers cannot allow
// that: applications that own all device memory through their own pool and
// forbid third-party allocations, and code that must not trigger the
// implicit device synchronisation of cudaMalloc/cudaFree inside a real-time
// loop.
// tf_pcg_jacobi_noalloc serves them: the caller passes the CSR matrix, the
// right-hand side and the solution in device memory; every other buffer the
// solve needs lives in one file-scope device array of fixed size
// (g_noalloc_scratch), which every GPU that loads the library holds until the
// process exits.  The call allocates nothing.
//
// The array is shared by all calls: calls that overlap on the GPU (two
// streams, two host threads) race on it and must be serialised by the caller.
// Each call clears the words that must start at zero (barrier counters, status)
// and writes every work vector before reading it.
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "krylov_dev.cuh"

namespace {

using tf::GridAR;
using tf::PackedAR;
using tf::PkState;

// control words, words of the packed reductions, the partials of grid_allreduce, work vectors r, z, p0, p1, q,
// 1 / diag (6 per row)
constexpr int kThreads = 512;
constexpr int kMaxBlocks = tf::kPkMaxBlocks;
constexpr int64_t kCtrlDoubles = 64;
constexpr int64_t kWordDoubles = 2 * 2 * tf::kPkWords;
constexpr int64_t kPartDoubles = 2 * (int64_t)kMaxBlocks * tf::kArMax;
constexpr int64_t kScratchDoubles = kCtrlDoubles + kWordDoubles + kPartDoubles + 6 * (int64_t)TF_NOALLOC_MAX_ROWS;

static __device__ __align__(256) double g_noalloc_scratch[kScratchDoubles];

// per-device address of g_noalloc_scratch (host code may not name the array
// itself: its host-side name is only a stand-in for the symbol)
double* g_scratch_ptr[64] = {};
std::mutex g_setup_mutex;

int scratch_for_current_device(double** out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return TF_ERR_NO_DEVICE;
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    if (!g_scratch_ptr[dev]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return TF_ERR_CUDA;
        g_scratch_ptr[dev] = (double*)p;
    }
    *out = g_scratch_ptr[dev];
    return TF_OK;
}

struct Ctrl {
    unsigned long long count;
    int status, iters;
    double resid;
    int converged;
    int nnz, longest;  // k_longest_row
};

// block 0 publishes the outcome of the solve (every exit path calls this)
__device__ void finish(Ctrl* ctl, int iters, double resid, bool converged) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        ctl->iters = iters;
        ctl->resid = resid;
        ctl->converged = converged ? 1 : 0;
    }
}

// ---- persistent PCG on CSR, G lanes per row ---------------------------------------
struct Args {
    int64_t m;
    const int32_t* rowptr;
    const int32_t* colind;
    const double* vals;
    const double* b;
    double* x;
    double* scratch;
    int max_iter;
    double tol;
    int rel;
};

constexpr int kInFlight = 8;   // entries a lane has in flight
constexpr int kFarTrips = 16;  // a row of more trips than this (128 entries on one lane) is summed by its warp
constexpr int far_length(int lanes) { return kFarTrips * kInFlight * lanes; }

// a lane's part of a row: every L-th entry from k
template <int L, class A, class LOAD, class TERM>
__device__ __forceinline__ A entries(const Args& a, A acc, int64_t row, int32_t k, int32_t e, LOAD load, TERM term) {
    constexpr int U = kInFlight;
    for (; k < e; k += U * L) {
        int32_t c[U];
        double v[U];
        decltype(load(0)) x[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool in = k + u * L < e;
            c[u] = in ? __ldg(a.colind + k + u * L) : 0;
            v[u] = in ? __ldg(a.vals + k + u * L) : 0.;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (k + u * L < e) x[u] = load(c[u]);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (k + u * L < e) acc = term(acc, row, c[u], v[u], x[u]);
    }
    return acc;
}
struct RowAndDiag {
    double sum, diag;
};
template <int L>
__device__ __forceinline__ void lanes_sum(double& v) {
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, L);
}
template <int L>
__device__ __forceinline__ void lanes_sum(RowAndDiag& v) {
    lanes_sum<L>(v.sum);
    lanes_sum<L>(v.diag);
}

// The rows go round-robin over the blocks, a warp's share at a time (small systems
// use every SM); a lane keeps eight entries in flight.  p = z + beta p is formed in
// the gathers, so an iteration has two grid steps, both packed integer reductions
// (krylov_dev.cuh).  Bound by latency below some 20,000 rows (two reductions, about
// 3 us, and the dependent trips to L2), by the FP64 pipe above: 21 instructions per
// row of a 7-point matrix on one lane, where G = 8 lanes issued their butterfly sums
// for 4 rows at a time.  Per iteration of a 7-point matrix, call included: 512 rows
// 16.1 -> 8.5 us, 8,000 23.0 -> 8.8, 65,231 34.4 -> 10.7, 238,328 70.4 -> 20.1 (before: 8
// lanes per row, up to 8 blocks of 256 per SM, counter barriers and FP64 tree sums).
//
// A matrix with rows of more than far_length(G) entries (bordered systems: a constraint, a Lagrange multiplier) takes the
// form that gives such a row to all lanes of its warp; on one lane every block waits for it.  With one dense row and
// column, us per iteration, one lane / the warp: 65,536 rows of 3 entries 8,192 / 339, 20,000 of 7 2,567 / 112, 20,000 of 41
// (8 lanes) 392 / 121.  The other matrices would pay 3 to 5% for the test in every product, k_longest_row costs them 3 us.
template <int G, bool FAR>
__global__ void __launch_bounds__(kThreads, 1) k_pcg_noalloc(Args a) {
    const int64_t m = a.m;
    Ctrl* ctl = reinterpret_cast<Ctrl*>(a.scratch);
    unsigned long long* const words = reinterpret_cast<unsigned long long*>(a.scratch + kCtrlDoubles);
    const GridAR g{&ctl->count, nullptr, a.scratch + kCtrlDoubles + kWordDoubles, &ctl->status};
    const PackedAR pa{words, &ctl->status}, pb{words + 2 * tf::kPkWords, &ctl->status};
    PkState ka, kb;
    unsigned long long epoch = 0;
    double* r = a.scratch + kCtrlDoubles + kWordDoubles + kPartDoubles;
    double* z = r + m;
    double* p0 = z + m;
    double* p1 = p0 + m;
    double* q = p1 + m;
    double* d = q + m;
    const int lane = threadIdx.x & 31, sub = lane & (G - 1);
    const int64_t first = ((threadIdx.x >> 5) * (int64_t)gridDim.x + blockIdx.x) * (32 / G) + lane / G;
    const int64_t step = (int64_t)gridDim.x * kThreads / G;
    __shared__ double sh[3];

    // sum over the entries of a row of term(row, column, value, load(column)), all lanes of the warp; FAR: the rows far above
    // the mean one after the other by the whole warp
    auto row_sum = [&](int64_t row, auto zero, auto load, auto term) {
        int32_t s = 0, e = 0;
        if (row < m) {
            s = __ldg(a.rowptr + row);
            e = __ldg(a.rowptr + row + 1);
        }
        const bool far = FAR && e - s > far_length(G);
        auto acc = entries<G>(a, zero, row, s + sub, far ? s : e, load, term);
        lanes_sum<G>(acc);
        if constexpr (FAR) {
            for (unsigned todo = __ballot_sync(0xffffffffu, far && sub == 0); todo; todo &= todo - 1u) {
                const int src = __ffs((int)todo) - 1;
                const int64_t fr = __shfl_sync(0xffffffffu, row, src);
                const int32_t fs = __shfl_sync(0xffffffffu, s, src), fe = __shfl_sync(0xffffffffu, e, src);
                auto w = entries<32>(a, zero, fr, fs + lane, fe, load, term);
                lanes_sum<32>(w);
                if (lane / G == src / G) acc = w;
            }
        }
        return acc;
    };
    const int64_t rounds = (m + step - 1) / step;  // the warps of a block make the same number of passes

    // diagonal (row scan, SolveGSstep<PB_JAC0>), r = b - A x, z = r/d, p0 = z
    {
        double v[3] = {0., 0., 0.};
        for (int64_t k = 0; k < rounds; ++k) {
            const int64_t row = first + k * step;
            const RowAndDiag t = row_sum(
                row, RowAndDiag{0., 0.}, [&](int32_t c) { return __ldcg(a.x + c); },
                [](const RowAndDiag& s, int64_t rw, int32_t c, double av, double x) {
                    return RowAndDiag{s.sum + av * x, c == rw ? av : s.diag};
                });
            if (sub == 0 && row < m) {
                const double bi = a.b[row], ri = bi - t.sum, di = 1.0 / t.diag, zi = ri * di;
                d[row] = di;
                r[row] = ri;
                z[row] = zi;
                p0[row] = zi;
                v[0] += ri * ri;
                v[1] += bi * bi;
                v[2] += zi * ri;
            }
        }
        double o[3];
        if (!tf::grid_allreduce<double, 3>(g, epoch, v, o)) return;
        if (threadIdx.x == 0) {
            double nb = sqrt(o[1]);
            if (nb == 0.0 || !a.rel) nb = 1.0;
            sh[0] = nb;
            sh[1] = sqrt(o[0]) / nb;
            sh[2] = o[2];
        }
        __syncthreads();
    }
    const double normb = sh[0];
    double resid = sh[1], rho = sh[2], beta = 0.;
    if (resid <= a.tol || a.max_iter == 0) {
        finish(ctl, 0, resid, resid <= a.tol);
        return;
    }
    struct Pair {
        double z, p;
    };
    double* pc = p0;
    double* pn = p1;
    for (int it = 1; it <= a.max_iter; ++it) {
        {
            double v[1] = {0.}, o[1];
            for (int64_t k = 0; k < rounds; ++k) {
                const int64_t row = first + k * step;
                const double acc = row_sum(
                    row, 0., [&](int32_t c) { return Pair{__ldcg(z + c), __ldcg(pc + c)}; },
                    [&](double s, int64_t, int32_t, double av, const Pair& x) { return s + av * (x.z + beta * x.p); });
                if (sub == 0 && row < m) {
                    const double pi = __ldcg(z + row) + beta * __ldcg(pc + row);
                    pn[row] = pi;
                    q[row] = acc;
                    v[0] += acc * pi;
                }
            }
            if (!tf::packed_allreduce<1>(pa, ka, g, epoch, v, o, false)) return;
            if (threadIdx.x == 0) sh[0] = rho / o[0];
            __syncthreads();
        }
        const double alpha = sh[0];
        {
            // the rows of the product, by the same threads
            double v[2] = {0., 0.}, o[2];
            for (int64_t k = 0; k < rounds; ++k) {
                const int64_t row = first + k * step;
                if (sub == 0 && row < m) {
                    a.x[row] += alpha * pn[row];
                    const double ri = r[row] - alpha * q[row];
                    const double zi = ri * d[row];
                    r[row] = ri;
                    z[row] = zi;
                    v[0] += ri * ri;
                    v[1] += zi * ri;
                }
            }
            if (!tf::packed_allreduce<2>(pb, kb, g, epoch, v, o, true)) return;
            if (threadIdx.x == 0) {
                sh[1] = sqrt(o[0]) / normb;
                sh[2] = o[1];
                sh[0] = o[1] / rho;
            }
            __syncthreads();
        }
        resid = sh[1];
        if (resid <= a.tol || it == a.max_iter) {
            finish(ctl, it, resid, resid <= a.tol);
            return;
        }
        rho = sh[2];
        beta = sh[0];
        double* t = pc;
        pc = pn;
        pn = t;
    }
}

__global__ void k_longest_row(int64_t m, const int32_t* __restrict__ rowptr, Ctrl* ctl) {
    int n = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
        n = max(n, rowptr[i + 1] - rowptr[i]);
    n = __reduce_max_sync(0xffffffffu, n);
    if ((threadIdx.x & 31) == 0 && n > 0) atomicMax(&ctl->longest, n);
    if (blockIdx.x == 0 && threadIdx.x == 0) ctl->nnz = rowptr[m];
}

}  // namespace

extern "C" int tf_pcg_jacobi_noalloc(int64_t m, const int32_t* rowptr, const int32_t* colind, const double* vals,
                                     const double* b, double* x, int* max_iter, double* tol, int rel, void* stream) {
    if (m <= 0 || !rowptr || !colind || !vals || !b || !x || !max_iter || !tol || *max_iter < 0) return TF_ERR_BAD_INPUT;
    if (m > TF_NOALLOC_MAX_ROWS) return TF_ERR_CAPACITY;
    double* scratch = nullptr;
    int st = scratch_for_current_device(&scratch);
    if (st != TF_OK) return st;
    cudaStream_t s = (cudaStream_t)stream;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return TF_ERR_CUDA;
    if (sms > kMaxBlocks) sms = kMaxBlocks;
    // the control words must start at zero; everything else is written before it is read
    if (cudaMemsetAsync(scratch, 0, sizeof(double) * (kCtrlDoubles + kWordDoubles), s) != cudaSuccess) return TF_ERR_CUDA;
    // average row length picks the lanes per row, the longest row their form; the matrix's row pointers are on the device
    Ctrl ctl;
    const int64_t scan = (m + 1023) / 1024;
    void* scan_args[] = {&m, &rowptr, &scratch};
    if (cudaLaunchKernel((const void*)k_longest_row, dim3((unsigned)(scan < sms ? scan : sms)), dim3(1024), scan_args, 0, s) !=
            cudaSuccess ||
        cudaMemcpyAsync(&ctl, scratch, sizeof(Ctrl), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return TF_ERR_CUDA;
    const double avg = (double)ctl.nnz / (double)m;
    // long rows are spread over lanes; 152 x 512 lanes hold 77,824 rows
    const int G = avg <= 32 ? 1 : avg <= 128 ? 8 : 32;
    const bool far = ctl.longest > far_length(G);
    const void* fn = G == 1   ? (far ? (const void*)k_pcg_noalloc<1, true> : (const void*)k_pcg_noalloc<1, false>)
                     : G == 8 ? (far ? (const void*)k_pcg_noalloc<8, true> : (const void*)k_pcg_noalloc<8, false>)
                              : (const void*)k_pcg_noalloc<32, false>;
    // at least four warps per block
    const int64_t want = (m * G + 127) / 128;
    int blocks = (int)(want < sms ? want : sms);
    if (blocks < 1) blocks = 1;
    Args a{m, rowptr, colind, vals, b, x, scratch, *max_iter, *tol, rel};
    void* args[] = {&a};
    if (cudaLaunchCooperativeKernel(fn, blocks, kThreads, args, 0, s) != cudaSuccess) return TF_ERR_CUDA;
    if (cudaMemcpyAsync(&ctl, scratch, sizeof(Ctrl), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return TF_ERR_CUDA;
    if (ctl.status != 0) return ctl.status;
    *max_iter = ctl.iters;
    *tol = ctl.resid;
    return ctl.converged ? TF_OK : TF_ERR_NOT_CONVERGED;
}

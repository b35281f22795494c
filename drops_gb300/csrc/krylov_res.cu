// Single-barrier Jacobi-PCG with each block's share of the system resident in
// shared memory (PCG of num/krylovsolver.h:107-189 in the Chronopoulos-Gear
// form of k_pcg_cg1, krylov.cu).
//
// k_pcg_cg1 waits on memory in every column step of its SELL walk: the
// column's 16-byte state {r, w, s, 1/d} is gathered through L1, and a warp's
// step lasts as long as its slowest lane, which often misses to L2.  Here
// block b owns the contiguous slot run [sb0, sb1) of the SELL matrix (equal
// column work, as in the blocked pass of k_pcg_cg1) for the whole solve, and
// a preprocessing kernel (once per pattern) lists the block's halo -- the
// rows of other blocks that its columns reference -- and translates each
// column of the run to a 16-bit index into the block's vector: its own slots
// first, then its halo rows.  Shared memory holds the translated columns, the
// run's values (as many as fit), the state, p and the correction dx of the
// block's rows.  Every pass then
//   1. forms u = (r - alpha (w + beta s)) / d for the block's rows and, from
//      the state gathered once from global memory, for its halo rows, into one
//      array (the halo loads are issued first, in one round; states lie in slot
//      order and a halo list ascends, so neighbouring threads share sectors);
//   2. walks its SELL run entirely in shared memory (column, value, u);
//   3. updates its rows, publishes their new state to the global double
//      buffer for the other blocks' halos, and joins the grid all-reduce.
// The owner and every halo reader evaluate u with the same operations, so all
// blocks use bitwise the same vector.
//
// T = float: the mixed-precision solver (FP32 iterations, the FP32 correction
// folded into the FP64 iterate at each refinement, refinement when the FP32
// residual has dropped by a factor 0.2 (TF_PCG_REL_UPDATE), claims
// convergence or max_iter is reached;
// convergence is decided on the FP64 residual b - A x).
// T = double: the FP64 solver on the same structure (32-byte state, FP64
// dots); it refines only when the recursive residual claims convergence or at
// max_iter, and then confirms convergence on the true residual b - A x.  The
// precomputed u keeps it at one FP64 multiply-add per stored entry (the
// on-the-fly u of k_pcg_cg1 would cost three more on GB300's narrow FP64 pipe).
//
// Mixed, per iteration on GB300 (P2 sphere on 96^3 cubes, 146,042 rows): 12.4 us
// with the counter all-reduce, states in row order and p of the halo kept in
// shared memory; 11.3 us with the packed reduction and the room given to matrix
// values (a block whose last slices' values came from L2 walked 6.2 us instead of
// 4.4); 9.3 us with the states in slot order and ascending halo lists (the block
// with the largest halo loaded it in 2.6 us against 1.2 in the mean); 6.8 us with
// loads that are known to be shared (a pointer that may be either is a generic load:
// the product took 3.9 us, now 2.9), the warps' ranges kept, and without the last
// window's empty slices (one warp of the last block did them all while the others
// waited, 1.4 us).  The product is now bound by shared memory: 2.9 bank conflicts per
// gather, 5.4 cycles per 32 entries.
//
// Applicability is decided on the host: every block's run (slot rows, halo,
// translated columns) must fit the shared memory and its vector 16-bit
// indices; otherwise the caller uses k_pcg_cg1 / the two-barrier FP64 kernel.
#include "krylov_dev.cuh"

namespace tf {

namespace {

constexpr int kResThreads = 512;
constexpr int kHaloMax = 4096;    // halo rows per block
constexpr int kHashSlots = 8192;  // open-addressing table of the halo preprocessing

struct alignas(32) Dstate {
    double x, y, z, w;
};
template <class T>
struct ResState;
template <>
struct ResState<float> {
    using V = float4;
};
template <>
struct ResState<double> {
    using V = Dstate;
};

__device__ __forceinline__ float4 st_ld(const float4* p) { return __ldca(p); }
__device__ __forceinline__ Dstate st_ld(const Dstate* p) {
    const double2 a = __ldca(reinterpret_cast<const double2*>(p)), b = __ldca(reinterpret_cast<const double2*>(p) + 1);
    return Dstate{a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ void st_st(float4* p, float4 v) { *p = v; }
__device__ __forceinline__ void st_st(Dstate* p, Dstate v) {
    reinterpret_cast<double2*>(p)[0] = make_double2(v.x, v.y);
    reinterpret_cast<double2*>(p)[1] = make_double2(v.z, v.w);
}
__device__ __forceinline__ float4 mk_state(float r, float w, float s, float id) { return make_float4(r, w, s, id); }
__device__ __forceinline__ Dstate mk_state(double r, double w, double s, double id) { return Dstate{r, w, s, id}; }

__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// u_{i+1} of a row from its state {r_i, w_i, s_{i-1}, 1/d}; the owner's row
// update evaluates exactly this sequence
template <class T, class V>
__device__ __forceinline__ T res_u(const V& v, T al, T be) {
    const T s = fma_rn(be, v.z, v.y);
    const T r = fma_rn(-al, s, v.x);
    return mul_rn(r, v.w);
}

template <class T>
struct PcgResArgs {
    using V = typename ResState<T>::V;
    int64_t m, nslices;
    const int32_t* perm;
    const int32_t* ptr;
    const int32_t* col;
    const uint16_t* col_tr;    // SELL columns translated to the owning block's vector
    const int32_t* halo_slots;  // [block][kHaloMax]
    const int32_t* halo_n;     // [block]
    const T* val;              // SELL values in T
    const double* val64;       // SELL values in FP64 (true residual)
    const T* diag;
    const double* b;
    double* x;
    V* V0;
    V* V1;
    T* P;
    GridAR g;
    PackedAR pk;
    int max_iter;
    double tol;
    int rel;
    double rel_update;  // refine when the recursive residual dropped by this factor (0: never)
    int* out_iter;
    double* out_resid;
    int* out_updates;
    int smax;      // slices of the largest run: sizes the per-slot arrays
    int hmax;      // halo rows of the largest halo (a multiple of 8)
    int32_t ccap;  // translated column slots (>= the largest run, a multiple of 16)
    int32_t vcap;  // value slots kept in shared memory
};

// dynamic shared memory of one block, in this order (every part a multiple of 32 bytes):
// Vs[slots] state, Us[slots + hmax] u, Ps[slots] p, sdx[slots], wsm[slots], ssm[slots],
// sperm[slots], hrow[hmax], ccol[ccap] (16-bit), cval[vcap]
template <class T>
inline size_t res_fixed_bytes(int smax, int hmax, int32_t ccap) {
    using V = typename ResState<T>::V;
    const size_t slots = (size_t)smax * 32;
    return slots * (sizeof(V) + 5 * sizeof(T) + sizeof(int32_t)) + (size_t)hmax * (sizeof(T) + sizeof(int32_t)) +
           (((size_t)ccap * 2 + 31) & ~(size_t)31);
}

template <class T>
__global__ void __launch_bounds__(kResThreads, 1) k_pcg_res(PcgResArgs<T> a) {
    using V = typename ResState<T>::V;
    constexpr int NW = kResThreads / 32;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    extern __shared__ __align__(32) unsigned char res_dyn[];
    const size_t slots = (size_t)a.smax * 32;
    V* Vs = reinterpret_cast<V*>(res_dyn);
    T* Us = reinterpret_cast<T*>(Vs + slots);
    T* Ps = Us + slots + a.hmax;
    T* sdx = Ps + slots;
    T* wsm = sdx + slots;  // products A u; with ssm also the FP64 residual products
    T* ssm = wsm + slots;  // products A p (refresh)
    double* rres = reinterpret_cast<double*>(wsm);
    int32_t* sperm = reinterpret_cast<int32_t*>(ssm + slots);
    int32_t* hrow = sperm + slots;
    uint16_t* ccol = reinterpret_cast<uint16_t*>(hrow + a.hmax);
    T* cval = reinterpret_cast<T*>(reinterpret_cast<unsigned char*>(ccol) + (((size_t)a.ccap * 2 + 31) & ~(size_t)31));
    __shared__ BalShared<NW, T> bsh;
    __shared__ BalShared<NW, double> bshd;
    __shared__ double sh[4];

    unsigned long long epoch = 0;
    PkState pk;
    V* Vc = a.V0;
    V* Vn = a.V1;
    const int64_t sb0 = balanced_part_start(a.ptr, a.nslices, blockIdx.x, gridDim.x);
    const int64_t sb1 = balanced_part_start(a.ptr, a.nslices, blockIdx.x + 1, gridDim.x);
    const int S = (int)(sb1 - sb0);
    const int NS = S * 32;  // own slots; halo entries follow at NS + h
    const int64_t NS0 = sb0 * 32;  // first own slot: states and p are published in slot order
    const int32_t pb = __ldg(a.ptr + sb0), pe = __ldg(a.ptr + sb1);
    const int32_t nslot = pe - pb;
    const int nh = __ldg(a.halo_n + blockIdx.x);
    // the run: slot rows, halo rows, translated columns, leading values; p = dx = 0
    for (int k = threadIdx.x; k < NS; k += kResThreads) {
        sperm[k] = __ldg(a.perm + sb0 * 32 + k);
        Ps[k] = T(0);
        sdx[k] = T(0);
    }
    for (int h = threadIdx.x; h < nh; h += kResThreads) hrow[h] = __ldg(a.halo_slots + (size_t)blockIdx.x * kHaloMax + h);
    for (int32_t k = threadIdx.x; k < nslot; k += kResThreads) {
        ccol[k] = __ldg(a.col_tr + pb + k);
        if (k < a.vcap) cval[k] = __ldg(a.val + pb + k);
    }
    sell_block_plan<NW, T>(bsh, a.ptr, sb0, S);
    sell_block_plan<NW, double>(bshd, a.ptr, sb0, S);  // ends with a block barrier
    __shared__ WalkRange wrs[NW];
    if (lane == 0) wrs[wid] = sell_block_range(bsh, S);
    __syncwarp();

    const int max_iter = a.max_iter;
    const double tol = a.tol;
    double normb = 1.0;
    int it = 0, updates = 0;
    bool converged = false;
    T gam = T(0), alpha = T(0), beta = T(0), thr_rel = T(0), thr_tol = T(0);

    // r = b - A x in FP64 over the block's rows (first: state {r, 0, 0, 1/d}, p = 0)
    auto true_residual = [&](bool first, bool& done) -> bool {
        const double* x = a.x;
        sell_block_walk<NW, double>(bshd, a.ptr, a.col, a.val64, sb0, S, [&](int32_t j) { return kld(x + j); },
                                    [&](int64_t s, double v) { rres[(s - sb0) * 32 + lane] = v; });
        double v[2] = {0., 0.};
        for (int i = wid; i < S; i += NW) {
            const int ls = i * 32 + lane;
            const int32_t row = sperm[ls];
            if (row >= 0) {
                const double bi = a.b[row];
                const double ri = bi - rres[ls];
                V vc;
                if (first) {
                    vc = mk_state((T)ri, T(0), T(0), T(1) / a.diag[row]);
                    a.P[NS0 + ls] = T(0);
                } else {
                    vc = Vs[ls];
                    vc.x = (T)ri;
                }
                Vs[ls] = vc;
                st_st(Vc + NS0 + ls, vc);
                v[0] += ri * ri;
                if (first) v[1] += bi * bi;
            }
        }
        double o[2];
        if (!grid_allreduce<double, 2>(a.g, epoch, v, o)) return false;
        if (threadIdx.x == 0) {
            double nb = normb;
            if (first) {
                nb = sqrt(o[1]);
                if (nb == 0.0 || !a.rel) nb = 1.0;
            }
            const double rl = sqrt(o[0]);
            sh[0] = nb;
            sh[1] = rl;
            sh[2] = rl / nb;
        }
        __syncthreads();
        normb = sh[0];
        const double r_last = sh[1], resid = sh[2];
        __syncthreads();
        ++updates;
        converged = resid <= tol;
        done = converged || it >= max_iter;
        thr_rel = (T)(a.rel_update * r_last);
        thr_tol = (T)(tol * normb);
        if (blockIdx.x == 0 && threadIdx.x == 0) *a.out_resid = resid;
        return true;
    };

    // one SpMV pass over the block's run; refresh: w = A (r / d) and s = A p
    // with r, p kept (after a true residual), else the CG step with (alpha, beta)
    auto pass = [&](bool refresh, T (&o)[6]) -> bool {
        T v[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
        const T al = refresh ? T(0) : alpha, be = refresh ? T(0) : beta;
        // u of the block's rows and of its halo: the halo states (global memory) are loaded first,
        // kHaloRegs per thread at once, and the block's own rows (shared memory) are done while they
        // are in flight (fewer at once for the 32-byte FP64 state: registers)
        constexpr int kHaloRegs = sizeof(T) == 4 ? 4 : 2;
        V hv[kHaloRegs];
#pragma unroll
        for (int q = 0; q < kHaloRegs; ++q) {
            const int h = threadIdx.x + q * kResThreads;
            if (h < nh) hv[q] = st_ld(Vc + hrow[h]);
        }
        for (int t = threadIdx.x; t < NS; t += kResThreads) Us[t] = sperm[t] >= 0 ? res_u<T>(Vs[t], al, be) : T(0);
#pragma unroll
        for (int q = 0; q < kHaloRegs; ++q) {
            const int h = threadIdx.x + q * kResThreads;
            if (h < nh) Us[NS + h] = res_u<T>(hv[q], al, be);
        }
        for (int h = threadIdx.x + kHaloRegs * kResThreads; h < nh; h += kResThreads)
            Us[NS + h] = res_u<T>(st_ld(Vc + hrow[h]), al, be);
        __syncthreads();
        // the slice offsets of the run come from the plan in shared memory:
        // ptr[sb0 + i] - pb = 32 * bsh.P[i]
        auto walk = [&](auto emit) {
            sell_block_walk_range(
                bsh, sb0, S, wrs[wid],
                [&](int64_t s, int32_t c0, int32_t n) {
                    const int i = (int)(s - sb0);
                    const int32_t p0 = 32 * (bsh.P[i] + c0) + lane;
                    const bool vsh = 32 * bsh.P[i + 1] <= a.vcap;
                    return vsh ? res_row<true, T>(ccol + p0, cval + p0, n, Us)
                               : res_row<false, T>(ccol + p0, a.val + pb + p0, n, Us);
                },
                [&](int64_t s, T val) { emit((int)(s - sb0) * 32 + lane, val); });
        };
        // row update of one slot from its product w = A u (refresh: and s = A p)
        auto row_update = [&](int ls, T wn, T sx) {
            if (sperm[ls] < 0) return;
            const V vc = Vs[ls];
            T sn, rn, pn;
            if (refresh) {
                sn = sx;
                rn = vc.x;
                pn = Ps[ls];
            } else {
                sn = fma_rn(be, vc.z, vc.y);
                rn = fma_rn(-al, sn, vc.x);
                pn = fma_rn(be, Ps[ls], mul_rn(vc.x, vc.w));
                Ps[ls] = pn;
                sdx[ls] = fma_rn(al, pn, sdx[ls]);
            }
            const T un = mul_rn(rn, vc.w);
            const V nv = mk_state(rn, wn, sn, vc.w);
            Vs[ls] = nv;
            st_st(Vn + NS0 + ls, nv);
            v[0] += rn * un;
            v[1] += un * wn;
            v[2] += un * sn;
            v[3] += pn * wn;
            v[4] += pn * sn;
            v[5] += rn * rn;
        };
        if (!refresh) {
            walk([&](int ls, T val) { wsm[ls] = val; });
            for (int i = wid; i < S; i += NW) row_update(i * 32 + lane, wsm[i * 32 + lane], T(0));
        } else {
            // w = A u, then s = A p recomputed, ending the drift of its recurrence
            walk([&](int ls, T val) { wsm[ls] = val; });
            for (int t = threadIdx.x; t < NS; t += kResThreads) Us[t] = Ps[t];
            for (int h = threadIdx.x; h < nh; h += kResThreads) Us[NS + h] = kld(a.P + hrow[h]);
            __syncthreads();
            walk([&](int ls, T val) { ssm[ls] = val; });
            for (int i = wid; i < S; i += NW) row_update(i * 32 + lane, wsm[i * 32 + lane], ssm[i * 32 + lane]);
        }
        if (!packed_allreduce<6>(a.pk, pk, a.g, epoch, v, o, true)) return false;
        V* t = Vc;
        Vc = Vn;
        Vn = t;
        return true;
    };

    // FP64 fold of the correction into x, p published for the refresh pass
    auto fold = [&]() -> bool {
        for (int i = wid; i < S; i += NW) {
            const int ls = i * 32 + lane;
            const int32_t row = sperm[ls];
            if (row >= 0) {
                a.x[row] += (double)sdx[ls];
                sdx[ls] = T(0);
                a.P[NS0 + ls] = Ps[ls];
            }
        }
        return grid_sync_ar(a.g, epoch);
    };

    bool done = false;
    if (!true_residual(true, done)) return;
    bool first = true;
    while (!done) {
        T o[6];
        if (!pass(true, o)) return;
        beta = first ? T(0) : o[0] / gam;
        first = false;
        gam = o[0];
        alpha = gam / (o[1] + beta * (o[2] + o[3]) + beta * beta * o[4]);
        bool refine = false;
        while (!refine) {
            if (!pass(false, o)) return;
            ++it;
            const T rn = sqrt(o[5]);
            refine = rn <= thr_rel || rn <= thr_tol || it >= max_iter;
            if (!refine) {
                beta = o[0] / gam;
                gam = o[0];
                alpha = gam / (o[1] + beta * (o[2] + o[3]) + beta * beta * o[4]);
            }
        }
        if (!fold()) return;
        if (!true_residual(false, done)) return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *a.out_iter = converged ? it : -1 - it;
        *a.out_updates = updates;
    }
}

// ---------------------------------------------------------------------------
// FP64 PCG with the reference's recurrences on the resident structure
// (PCGSolverCL<JACPcCL>::Solve, num/krylovsolver.h:107-189): two reductions per
// iteration, <p, A p> and then <r, r>, <z, r>.  A block keeps its rows' p, r, x
// and 1/d, its translated columns and its values in shared memory, and its own
// copy of the halo rows' p, which it advances itself (p = z + beta p) from the
// owners' published z: one 8-byte load per halo row and iteration, one FP64
// multiply-add per stored entry, no division in the row updates.
//
// Bound: latency of the two reductions and the FP64 pipe (64 cycles per warp
// instruction and quarter of an SM).  Against the kernel that walks the SELL
// matrix in global memory and forms z + beta p per entry (k_pcg, which remains
// for systems whose block share does not fit), per iteration on GB300:
// P2 torus on 41^3 cubes (35,592 rows, 152 blocks) 23.1 -> 9.6 us, P1 sphere on
// 16^3 (664 rows, 16 blocks) 12.1 -> 8.4 us.
// ---------------------------------------------------------------------------
struct Pcg64Args {
    int64_t m, nslices;
    const int32_t* perm;
    const int32_t* ptr;
    const uint16_t* col_tr;
    const int32_t* halo_slots;
    const int32_t* halo_n;
    const double* val;
    const double* diag;
    const double* b;
    double* x;
    double* Z;
    GridAR g;
    PackedAR pk1, pk2;
    int max_iter;
    double tol;
    int rel;
    int* out_iter;
    double* out_resid;
    int smax, hmax;
    int32_t ccap, vcap;
};

// dynamic shared memory: Ps[slots + hmax] p, rs, xs, ds, qs[slots] each, sperm[slots], hrow[hmax],
// ccol[ccap] (16-bit), cval[vcap]
inline size_t pcg64_fixed_bytes(int smax, int hmax, int32_t ccap) {
    const size_t slots = (size_t)smax * 32;
    return slots * (5 * sizeof(double) + sizeof(int32_t)) + (size_t)hmax * (sizeof(double) + sizeof(int32_t)) +
           (((size_t)ccap * 2 + 31) & ~(size_t)31);
}

__global__ void __launch_bounds__(kResThreads, 1) k_pcg64_res(Pcg64Args a) {
    constexpr int NW = kResThreads / 32;
    const int lane = threadIdx.x & 31;
    extern __shared__ __align__(32) unsigned char res_dyn[];
    const size_t slots = (size_t)a.smax * 32;
    double* Ps = reinterpret_cast<double*>(res_dyn);
    double* rs = Ps + slots + a.hmax;
    double* xs = rs + slots;
    double* ds = xs + slots;  // 1 / diagonal
    double* qs = ds + slots;
    int32_t* sperm = reinterpret_cast<int32_t*>(qs + slots);
    int32_t* hrow = sperm + slots;
    uint16_t* ccol = reinterpret_cast<uint16_t*>(hrow + a.hmax);
    double* cval = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(ccol) + (((size_t)a.ccap * 2 + 31) & ~(size_t)31));
    __shared__ BalShared<NW, double> bsh;
    __shared__ double sh[4];  // alpha, beta, 1 / rho, rho
    __shared__ int flag, conv;

    unsigned long long epoch = 0;
    PkState pk1, pk2;
    const int64_t sb0 = balanced_part_start(a.ptr, a.nslices, blockIdx.x, gridDim.x);
    const int64_t sb1 = balanced_part_start(a.ptr, a.nslices, blockIdx.x + 1, gridDim.x);
    const int S = (int)(sb1 - sb0), NS = S * 32;
    const int32_t pb = __ldg(a.ptr + sb0), nslot = __ldg(a.ptr + sb1) - pb;
    const int nh = __ldg(a.halo_n + blockIdx.x);
    for (int k = threadIdx.x; k < NS; k += kResThreads) {
        const int32_t row = __ldg(a.perm + sb0 * 32 + k);
        sperm[k] = row;
        const double x = row >= 0 ? a.x[row] : 0.;
        xs[k] = x;
        Ps[k] = x;  // operand of the first product
        ds[k] = row >= 0 ? 1.0 / a.diag[row] : 0.;
    }
    for (int h = threadIdx.x; h < nh; h += kResThreads) {
        const int32_t slot = __ldg(a.halo_slots + (size_t)blockIdx.x * kHaloMax + h);
        hrow[h] = slot;
        Ps[NS + h] = a.x[__ldg(a.perm + slot)];
    }
    for (int32_t k = threadIdx.x; k < nslot; k += kResThreads) {
        ccol[k] = __ldg(a.col_tr + pb + k);
        if (k < a.vcap) cval[k] = __ldg(a.val + pb + k);
    }
    sell_block_plan<NW, double>(bsh, a.ptr, sb0, S);  // ends with a block barrier
    __shared__ WalkRange wrs[NW];
    if (lane == 0) wrs[threadIdx.x >> 5] = sell_block_range(bsh, S);
    __syncwarp();
    // q = A Ps over the run; returns this thread's part of <q, Ps>
    auto walk = [&]() -> double {
        double pq = 0.;
        sell_block_walk_range(
            bsh, sb0, S, wrs[threadIdx.x >> 5],
            [&](int64_t s, int32_t c0, int32_t n) {
                const int i = (int)(s - sb0);
                const int32_t p0 = 32 * (bsh.P[i] + c0) + lane;
                const bool vsh = 32 * bsh.P[i + 1] <= a.vcap;
                return vsh ? res_row<true, double>(ccol + p0, cval + p0, n, Ps)
                           : res_row<false, double>(ccol + p0, a.val + pb + p0, n, Ps);
            },
            [&](int64_t s, double val) {
                const int ls = (int)(s - sb0) * 32 + lane;
                qs[ls] = val;
                pq += val * Ps[ls];
            });
        return pq;
    };
    double thr2, normb, rr;
    int it = 0;
    {
        walk();
        double v[3] = {0., 0., 0.};
        for (int t = threadIdx.x; t < NS; t += kResThreads) {
            const int32_t row = sperm[t];
            double r = 0., z = 0.;
            if (row >= 0) {
                const double bi = a.b[row];
                r = bi - qs[t];
                z = r * ds[t];
                v[1] += bi * bi;
            }
            a.Z[sb0 * 32 + t] = z;
            rs[t] = r;
            Ps[t] = 0.;
            v[0] += r * r;
            v[2] += z * r;
        }
        for (int h = threadIdx.x; h < nh; h += kResThreads) Ps[NS + h] = 0.;
        double o[3];
        if (!grid_allreduce<double, 3>(a.g, epoch, v, o)) return;
        double nb = 1.0;
        if (threadIdx.x == 0) {
            nb = sqrt(o[1]);
            if (nb == 0.0 || !a.rel) nb = 1.0;
            sh[0] = nb;
            sh[1] = 0.;
            sh[2] = 1.0 / o[2];
            sh[3] = o[2];
            conv = rr_reached(o[0], rr_threshold(a.tol, nb), a.tol, nb);
            flag = conv || a.max_iter <= 0;
        }
        rr = o[0];
        __syncthreads();
        normb = sh[0];
        thr2 = rr_threshold(a.tol, normb);
    }
    bool done = flag != 0;
    while (!done) {
        const double beta = sh[1];
        // p = z + beta p on the halo and the block's rows
        for (int h = threadIdx.x; h < nh; h += kResThreads) Ps[NS + h] = __ldcg(a.Z + hrow[h]) + beta * Ps[NS + h];
        for (int t = threadIdx.x; t < NS; t += kResThreads) Ps[t] = rs[t] * ds[t] + beta * Ps[t];
        __syncthreads();
        double v1[1], o1[1];
        v1[0] = walk();
        if (!packed_allreduce<1>(a.pk1, pk1, a.g, epoch, v1, o1, false)) return;
        if (threadIdx.x == 0) sh[0] = rho_by(sh[3], sh[2], o1[0]);  // alpha = rho / <p, A p>
        __syncthreads();
        const double alpha = sh[0];
        double v[2] = {0., 0.}, o[2];
        for (int t = threadIdx.x; t < NS; t += kResThreads) {
            xs[t] += alpha * Ps[t];
            const double r = rs[t] - alpha * qs[t];
            const double z = r * ds[t];
            rs[t] = r;
            a.Z[sb0 * 32 + t] = z;
            v[0] += r * r;
            v[1] += z * r;
        }
        if (!packed_allreduce<2>(a.pk2, pk2, a.g, epoch, v, o, true)) return;
        ++it;
        rr = o[0];
        if (threadIdx.x == 0) {
            sh[1] = by_rho(o[1], sh[3], sh[2]);
            sh[3] = o[1];
            conv = rr_reached(rr, thr2, a.tol, normb);
            flag = conv || it >= a.max_iter;
        }
        __syncthreads();
        // 1 / rho of the next iteration, off the path of the others (read after two barriers)
        if (threadIdx.x == kResThreads - 32) sh[2] = 1.0 / o[1];
        done = flag != 0;
    }
    for (int t = threadIdx.x; t < NS; t += kResThreads)
        if (sperm[t] >= 0) a.x[sperm[t]] = xs[t];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *a.out_iter = conv ? it : -1 - it;
        *a.out_resid = sqrt(rr) / normb;
    }
}

__global__ void k_res_diag32(int64_t n, const double* __restrict__ a, float* __restrict__ b) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        b[i] = (float)a[i];
}

__global__ void k_sell_iperm(int64_t nslots, const int32_t* __restrict__ perm, int32_t* __restrict__ iperm) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nslots; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t r = perm[i];
        if (r >= 0) iperm[r] = (int32_t)i;
    }
}

// Per part b of the balanced partition (one block each): the halo slots (the
// distinct columns of the run, as slots, that lie outside it), ascending, so
// that consecutive threads read neighbouring states, and the run's columns
// translated to the block's vector (own slot, or NS + halo number).  An open-
// addressing table finds the distinct ones, a bitonic sort orders them, a
// binary search translates.  info[0]: set when a table or a halo overflows or an
// index needs more than 16 bits; info[1]: largest run in slices, info[2]: largest
// run in slots, info[3]: largest halo.
__device__ __forceinline__ uint32_t halo_hash(int32_t c) { return ((uint32_t)c * 2654435761u) >> 19; }  // 13 bits
static_assert(kHashSlots == 1 << 13, "hash width");

__global__ void __launch_bounds__(512) k_res_halo(const int32_t* __restrict__ ptr, int64_t nslices,
                                                  const int32_t* __restrict__ col, const int32_t* __restrict__ iperm,
                                                  uint16_t* __restrict__ col_tr, int32_t* __restrict__ halo_slots,
                                                  int32_t* __restrict__ halo_n, int* __restrict__ info) {
    extern __shared__ int32_t hsh[];  // keys[kHashSlots], list[kHaloMax]
    int32_t* keys = hsh;
    int32_t* list = hsh + kHashSlots;
    __shared__ int bad, cnt;
    const int64_t sb0 = balanced_part_start(ptr, nslices, blockIdx.x, gridDim.x);
    const int64_t sb1 = balanced_part_start(ptr, nslices, blockIdx.x + 1, gridDim.x);
    const int NS = (int)(sb1 - sb0) * 32;
    const int32_t lo = (int32_t)(sb0 * 32), hi = (int32_t)(sb1 * 32);
    const int32_t pb = ptr[sb0], pe = ptr[sb1];
    for (int i = threadIdx.x; i < kHashSlots; i += blockDim.x) keys[i] = -1;
    if (threadIdx.x == 0) bad = cnt = 0;
    __syncthreads();
    for (int32_t k = pb + threadIdx.x; k < pe; k += blockDim.x) {
        const int32_t sl = iperm[col[k]];
        if (sl >= lo && sl < hi) continue;
        uint32_t h = halo_hash(sl);
        int probe = 0;
        for (; probe < kHashSlots; ++probe) {
            const int32_t old = atomicCAS(&keys[h], -1, sl);
            if (old == -1) {
                const int id = atomicAdd(&cnt, 1);  // the order is lost in the sort
                if (id < kHaloMax) list[id] = sl;
            }
            if (old == -1 || old == sl) break;
            h = (h + 1) & (kHashSlots - 1);
        }
        if (probe == kHashSlots) bad = 1;
    }
    __syncthreads();
    const int nh = cnt;
    if (threadIdx.x == 0 && (nh > kHaloMax || NS + nh > 65535)) bad = 1;
    __syncthreads();
    if (!bad) {
        int np = 1;
        while (np < nh) np <<= 1;  // at most kHaloMax
        for (int i = nh + threadIdx.x; i < np; i += blockDim.x) list[i] = 0x7fffffff;
        __syncthreads();
        for (int size = 2; size <= np; size <<= 1)
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int i = threadIdx.x; i < np; i += blockDim.x) {
                    const int p = i ^ stride;
                    if (p > i) {
                        const int32_t x = list[i], y = list[p];
                        if ((x > y) == ((i & size) == 0)) {
                            list[i] = y;
                            list[p] = x;
                        }
                    }
                }
                __syncthreads();
            }
        for (int i = threadIdx.x; i < nh; i += blockDim.x) halo_slots[(size_t)blockIdx.x * kHaloMax + i] = list[i];
        for (int32_t k = pb + threadIdx.x; k < pe; k += blockDim.x) {
            const int32_t sl = iperm[col[k]];
            int32_t tr = sl - lo;
            if (sl < lo || sl >= hi) {
                int l = 0, r = nh - 1;  // list[l] == sl at the end: inserted above
                while (l < r) {
                    const int mid = (l + r) >> 1;
                    if (list[mid] < sl) l = mid + 1;
                    else r = mid;
                }
                tr = NS + l;
            }
            col_tr[k] = (uint16_t)tr;
        }
    }
    if (threadIdx.x == 0) {
        halo_n[blockIdx.x] = nh;
        if (bad) atomicOr(info, 1);
        atomicMax(info + 1, (int)(sb1 - sb0));
        atomicMax(info + 2, pe - pb);
        atomicMax(info + 3, nh);
    }
}

int mat_slot(Context* c, const CSR& A) {
    for (int i = 0; i < TF_NUM_MATS; ++i)
        if (&c->mats[i] == &A) return i;
    return 0;
}

// halo lists and translated columns, once per pattern and grid
int ensure_res_plan(Context* c, CSR& A, int blocks) {
    Sell& S = A.sell;
    const int id = mat_slot(c, A);
    TF_TRY(ensure_sell_iperm(c, A));
    if (S.res_blocks != blocks) {
        TF_TRY(ensure(c, c->sell_coltr[id], (size_t)(S.npad > 0 ? S.npad : 1)));
        TF_TRY(ensure(c, c->sell_halo[id], (size_t)blocks * kHaloMax + blocks));
        S.col_tr = c->sell_coltr[id].p;
        S.halo_slots = c->sell_halo[id].p;
        S.halo_n = c->sell_halo[id].p + (size_t)blocks * kHaloMax;
        TF_TRY(ensure(c, c->kry_iters, 4));
        TF_CUDA(c, cudaMemsetAsync(c->kry_iters.p, 0, 4 * sizeof(int), c->stream));
        const size_t hsm = sizeof(int32_t) * (kHashSlots + kHaloMax);
        TF_CUDA(c, cudaFuncSetAttribute((const void*)k_res_halo, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hsm));
        k_res_halo<<<blocks, 512, hsm, c->stream>>>(S.ptr, S.used, S.col, S.iperm, S.col_tr, S.halo_slots, S.halo_n,
                                                    c->kry_iters.p);
        ++c->launches;
        TF_CUDA(c, cudaGetLastError());
        int h[4] = {0, 0, 0, 0};
        TF_CUDA(c, cudaMemcpyAsync(h, c->kry_iters.p, 4 * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
        TF_CUDA(c, cudaStreamSynchronize(c->stream));
        S.res_ok = h[0] == 0;
        S.res_smax = h[1];
        S.res_maxslots = h[2];
        S.res_hmax = (h[3] + 7) & ~7;
        S.res_blocks = blocks;
    }
    return TF_OK;
}

// Blocks of a resident solve: one per SM, and at least two slices each (a
// smaller share saves less than another block adds to the reductions).
int res_blocks(const Context* c, const CSR& A) {
    return (int)std::max<int64_t>(1, std::min<int64_t>(std::min(c->num_sms, kPkMaxBlocks), A.sell.used / 2));
}

}  // namespace

// row -> slot map of the SELL layout, once per pattern
int ensure_sell_iperm(Context* c, CSR& A) {
    Sell& S = A.sell;
    if (S.iperm_gen == S.pattern_gen && S.iperm) return TF_OK;
    const int id = mat_slot(c, A);
    TF_TRY(ensure(c, c->sell_iperm[id], (size_t)(A.m > 0 ? A.m : 1)));
    S.iperm = c->sell_iperm[id].p;
    k_sell_iperm<<<grid_for(c, S.nslices * 32), kBlock, 0, c->stream>>>(S.nslices * 32, S.perm, S.iperm);
    ++c->launches;
    TF_CUDA(c, cudaGetLastError());
    S.iperm_gen = S.pattern_gen;
    S.res_blocks = 0;  // its plan follows the old map
    return TF_OK;
}

// zeroed words for n packed reductions
int packed_words(Context* c, int n, unsigned long long** w) {
    const size_t words = (size_t)n * 2 * kPkWords;
    TF_TRY(ensure(c, c->kry_packed, words));
    TF_CUDA(c, cudaMemsetAsync(c->kry_packed.p, 0, sizeof(unsigned long long) * words, c->stream));
    *w = c->kry_packed.p;
    return TF_OK;
}

// Resident single-barrier PCG; *applied = false (nothing launched) when a
// block's run does not fit the shared memory.
template <class T>
int pcg_resident(Context* c, CSR& A, const double* b, double* x, int* max_iter, double* tol, int rel, bool* applied) {
    using V = typename ResState<T>::V;
    *applied = false;
    const int64_t m = A.m;
    const void* fn = (const void*)k_pcg_res<T>;
    const int blocks = res_blocks(c, A);
    TF_TRY(ensure_res_plan(c, A, blocks));
    const Sell& S = A.sell;
    if (!S.res_ok || S.res_smax <= 0 || S.res_smax > kBalMaxSlices) return TF_OK;
    int64_t room = 0;
    TF_TRY(max_dynamic_smem(c, fn, &room));
    const int32_t ccap = (S.res_maxslots + 15) & ~15;
    const int64_t fixed = (int64_t)res_fixed_bytes<T>(S.res_smax, S.res_hmax, ccap);
    if (fixed > room) return TF_OK;
    int32_t vcap = (int32_t)std::min<int64_t>((room - fixed) / (int64_t)sizeof(T), (int64_t)ccap) & ~7;
    if (c->pcg_res_vcap_kb >= 0)
        vcap = std::min<int32_t>(vcap, (int32_t)(((int64_t)c->pcg_res_vcap_kb * 1024 / (int64_t)sizeof(T)) & ~7));
    const size_t dyn = (size_t)fixed + (size_t)vcap * sizeof(T);
    int per_sm = 0;
    TF_CUDA(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kResThreads, dyn));
    if (per_sm < 1) return TF_OK;

    // workspace: V0, V1 (a state per slot each), p (per slot), T diagonal (m)
    const int64_t ns = S.nslices * 32;
    const T* diag = nullptr;
    V* V0 = nullptr;
    T* P = nullptr;
    if constexpr (sizeof(T) == 4) {
        TF_TRY(ensure(c, c->kry32, (size_t)(9 * ns + m)));
        float* base = c->kry32.p;
        k_res_diag32<<<grid_for(c, m), kBlock, 0, c->stream>>>(m, A.diag, base + 9 * ns);
        ++c->launches;
        V0 = reinterpret_cast<V*>(base);
        P = base + 8 * ns;
        diag = base + 9 * ns;
    } else {
        TF_TRY(ensure(c, c->kry64, (size_t)(9 * ns)));
        double* base = c->kry64.p;
        V0 = reinterpret_cast<V*>(base);
        P = base + 8 * ns;
        diag = A.diag;
    }
    const size_t part_d = (size_t)2 * blocks * kArMax;
    TF_TRY(ensure(c, c->kry_part, part_d + (part_d + 1) / 2 + 16));
    TF_TRY(ensure(c, c->kry_bar, 2));
    TF_TRY(ensure(c, c->kry_iters, 4));
    TF_TRY(ensure(c, c->kry_resid, 1));
    TF_CUDA(c, cudaMemsetAsync(c->kry_bar.p, 0, 2 * sizeof(unsigned), c->stream));
    TF_CUDA(c, cudaMemsetAsync(c->status.p, 0, 4 * sizeof(int), c->stream));
    unsigned long long* pw = nullptr;
    TF_TRY(packed_words(c, 1, &pw));
    PcgResArgs<T> g;
    g.pk = PackedAR{pw, c->status.p};
    g.m = m;
    g.nslices = S.used;
    g.perm = S.perm;
    g.ptr = S.ptr;
    g.col = S.col;
    g.col_tr = S.col_tr;
    g.halo_slots = S.halo_slots;
    g.halo_n = S.halo_n;
    if constexpr (sizeof(T) == 4) g.val = S.v32;
    else g.val = S.v64;
    g.val64 = S.v64;
    g.diag = diag;
    g.b = b;
    g.x = x;
    g.V0 = V0;
    g.V1 = V0 + ns;
    g.P = P;
    g.g.count = reinterpret_cast<unsigned long long*>(c->kry_bar.p);
    g.g.partd = c->kry_part.p;
    g.g.partf = reinterpret_cast<float*>(c->kry_part.p + part_d);
    g.g.status = c->status.p;
    g.max_iter = *max_iter;
    g.tol = *tol;
    g.rel = rel;
    g.rel_update = sizeof(T) == 4 ? c->pcg_rel_update : 0.0;
    g.out_iter = c->kry_iters.p;
    g.out_resid = c->kry_resid.p;
    g.out_updates = c->kry_iters.p + 1;
    g.smax = S.res_smax;
    g.hmax = S.res_hmax;
    g.ccap = ccap;
    g.vcap = vcap;
    void* args[] = {&g};
    TF_CUDA(c, cudaLaunchCooperativeKernel(fn, blocks, kResThreads, args, dyn, c->stream));
    ++c->launches;
    *applied = true;
    int it[2] = {0, 0};
    double res = 0;
    TF_CUDA(c, cudaMemcpyAsync(it, c->kry_iters.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    TF_CUDA(c, cudaMemcpyAsync(&res, c->kry_resid.p, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    int st = 0;
    TF_TRY(sync_status(c, &st));
    if (st) return set_err(c, st, "pcg (resident): grid barrier watchdog fired");
    c->last_refinements = it[1];
    *max_iter = it[0] >= 0 ? it[0] : -1 - it[0];
    *tol = res;
    return it[0] >= 0 ? TF_OK : set_err(c, TF_ERR_NOT_CONVERGED, "pcg: no convergence within max_iter");
}

template int pcg_resident<float>(Context*, CSR&, const double*, double*, int*, double*, int, bool*);
template int pcg_resident<double>(Context*, CSR&, const double*, double*, int*, double*, int, bool*);

// FP64 PCG (reference recurrences) on the resident structure; *applied = false
// (nothing launched) when a block's run does not fit the shared memory.
int pcg64_resident(Context* c, CSR& A, const double* b, double* x, int* max_iter, double* tol, int rel, bool* applied) {
    *applied = false;
    const int64_t m = A.m;
    const void* fn = (const void*)k_pcg64_res;
    const int blocks = res_blocks(c, A);
    int64_t room = 0;
    TF_TRY(max_dynamic_smem(c, fn, &room));
    // No run is smaller than the mean, so a mean that does not fit rules the system out before its plan: a kernel over the
    // matrix and a wait.
    const Sell& S = A.sell;
    const int64_t mean_slices = (S.used + blocks - 1) / blocks, mean_slots = (S.npad + blocks - 1) / blocks;
    if (mean_slices > kBalMaxSlices || (int64_t)pcg64_fixed_bytes((int)mean_slices, 0, (int32_t)mean_slots) > room) return TF_OK;
    TF_TRY(ensure_res_plan(c, A, blocks));
    if (!S.res_ok || S.res_smax <= 0 || S.res_smax > kBalMaxSlices) return TF_OK;
    const int32_t ccap = (S.res_maxslots + 15) & ~15;
    const int64_t fixed = (int64_t)pcg64_fixed_bytes(S.res_smax, S.res_hmax, ccap);
    if (fixed > room) return TF_OK;
    const int32_t vcap = (int32_t)std::min<int64_t>((room - fixed) / (int64_t)sizeof(double), (int64_t)ccap) & ~7;
    const size_t dyn = (size_t)fixed + (size_t)vcap * sizeof(double);
    int per_sm = 0;
    TF_CUDA(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kResThreads, dyn));
    if (per_sm < 1) return TF_OK;
    TF_TRY(ensure(c, c->kry64, (size_t)(S.nslices * 32)));
    const size_t part_d = (size_t)2 * blocks * kArMax;
    TF_TRY(ensure(c, c->kry_part, part_d + 16));
    TF_TRY(ensure(c, c->kry_bar, 2));
    TF_TRY(ensure(c, c->kry_iters, 4));
    TF_TRY(ensure(c, c->kry_resid, 1));
    TF_CUDA(c, cudaMemsetAsync(c->kry_bar.p, 0, 2 * sizeof(unsigned), c->stream));
    TF_CUDA(c, cudaMemsetAsync(c->status.p, 0, 4 * sizeof(int), c->stream));
    unsigned long long* pw = nullptr;
    TF_TRY(packed_words(c, 2, &pw));
    Pcg64Args g{};
    g.pk1 = PackedAR{pw, c->status.p};
    g.pk2 = PackedAR{pw + 2 * kPkWords, c->status.p};
    g.m = m;
    g.nslices = S.used;
    g.perm = S.perm;
    g.ptr = S.ptr;
    g.col_tr = S.col_tr;
    g.halo_slots = S.halo_slots;
    g.halo_n = S.halo_n;
    g.val = S.v64;
    g.diag = A.diag;
    g.b = b;
    g.x = x;
    g.Z = c->kry64.p;
    g.g.count = reinterpret_cast<unsigned long long*>(c->kry_bar.p);
    g.g.partd = c->kry_part.p;
    g.g.status = c->status.p;
    g.max_iter = *max_iter;
    g.tol = *tol;
    g.rel = rel;
    g.out_iter = c->kry_iters.p;
    g.out_resid = c->kry_resid.p;
    g.smax = S.res_smax;
    g.hmax = S.res_hmax;
    g.ccap = ccap;
    g.vcap = vcap;
    void* args[] = {&g};
    TF_CUDA(c, cudaLaunchCooperativeKernel(fn, blocks, kResThreads, args, dyn, c->stream));
    ++c->launches;
    *applied = true;
    int it = 0;
    double res = 0;
    TF_CUDA(c, cudaMemcpyAsync(&it, c->kry_iters.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    TF_CUDA(c, cudaMemcpyAsync(&res, c->kry_resid.p, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    int st = 0;
    TF_TRY(sync_status(c, &st));
    if (st) return set_err(c, st, "pcg: grid barrier watchdog fired");
    *max_iter = it >= 0 ? it : -1 - it;
    *tol = res;
    return it >= 0 ? TF_OK : set_err(c, TF_ERR_NOT_CONVERGED, "pcg: no convergence within max_iter");
}

}  // namespace tf

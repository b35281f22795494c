// Restarted GMRES with modified Gram-Schmidt in two grid steps per Arnoldi
// step, as one persistent cooperative kernel (num/krylovsolver.h:320-463).
//
// Modified Gram-Schmidt subtracts one projection after the other, and every
// coefficient is a dot over all rows: i + 1 grid-wide reductions in Arnoldi
// step i.  The same coefficients follow from one reduction.  With
// a_k = <w, v_k> of the unprojected w and L_kj = <v_k, v_j> (j < k) of the
// basis,
//   h_k = <w - sum_{j<k} h_j v_j, v_k> = a_k - sum_{j<k} L_kj h_j,
// a forward substitution with the unit lower triangle I + L, so the
// coefficients keep modified Gram-Schmidt's correction for the basis' loss of
// orthogonality (the inverse compact WY form of Swirydowicz, Langou, Ananthan,
// Yang and Thomas, "Low synchronization Gram-Schmidt and generalized minimal
// residual algorithms", 2021).  An Arnoldi step is
//   1. w = B v_i on the block's rows, dots of w and of v_i with every basis
//      vector (row i of L comes from the same read of the basis); reduction of
//      2 i + 2 values;
//   2. h by forward substitution in every block, w -= V h, |w|^2; reduction of
//      one value, which is also the barrier before others gather w; Givens
//      rotation and stopping test in every block on identical values.
// B is A P^{-1} (right, point or nodal 2x2 block Jacobi) or P^{-1} A (left),
// formed once per matrix in SELL order: no division and no preconditioner pass
// in the loop.
//
// The solve runs in slot space: basis vectors are stored in the order of the
// SELL slots and the columns are translated to slots, so a block's rows are
// contiguous in every basis vector.  Each block owns a contiguous run of
// slices, keeps its part of w and v_i in shared memory, and takes the dots one
// basis vector per warp over all its rows: one warp reduction per eight dots
// and block, instead of one per eight dots and 32 rows.
//
// V = double: the reference's solver (cycles of restart - 1 steps, stopping
// test on the rotated residual).  V = float: mixed precision; every cycle runs
// in FP32 until its residual estimate has dropped by 1e-5 (or to tol), and the
// residual b - A x and the update of x are FP64: one step of iterative
// refinement per cycle.
//
// Bound: latency (grid round trips, FP64 instructions in chains).  Per Arnoldi
// step on GB300, mean over a solve, before (one reduction per projection in
// FP64, CGS2 with three grid steps in FP32) and now: Cahn-Hilliard block system
// of the 128^3 torus (119,752 rows) in FP32 40.8 -> 15.6 us, of the 40^3 torus
// (11,928 rows) in FP64 153 -> 17.3 us.  With counter reductions it was 18.9 and 21.4:
// product 4.6, dots 2.8, reduction 4.6 (2.9 of it the wait), coefficients 1.0, update
// 2.5, norm 3.3; packed sums took 2.4 off (FP32), the head of B in shared memory,
// shared memory loads and kept warp ranges the rest.
#include <algorithm>
#include <cmath>

#include "krylov_dev.cuh"

namespace tf {

namespace {

constexpr int kLsThreads = 512;
constexpr int kLsWarps = kLsThreads / 32;
constexpr int kLsMaxR = 64;                 // restart length
constexpr int kLsVals = 2 * kLsMaxR + 8;    // values of one reduction, per block (at most 2 R)

template <class V>
struct GmLsArgs {
    int64_t nslices, m;
    const int32_t* perm;
    const int32_t* ptr;
    const int32_t* col;    // row numbering (residual)
    const int32_t* cols;   // slot numbering (Arnoldi products)
    const V* bval;         // B in SELL order
    const double* aval;    // A in SELL order
    const double* b;
    double* x;
    const double* diag;    // point Jacobi; nullptr with binv
    const double* binv;    // nodal 2x2 inverses [m/2][4]
    V* basis;              // (R + 1) x ld, unnormalised: v_k = scl[k] * basis_k
    int64_t ld;
    V* zrow;               // m values (block Jacobi: the update before P^{-1})
    V* part;               // [2][blocks][kLsVals]
    GridAR g;
    PackedAR pkd, pkn;     // dots, norm
    int R, max_iter, rel, left, nloc;  // nloc: slots of the largest run held in shared memory (0: none)
    int ccap;              // entries of the block's part of B kept in shared memory
    double tol, inner_floor;
    int* out_iter;
    double* out_resid;
    int* out_cycles;
};

template <class V>
struct LsSmall {  // least-squares state, identical in every block
    V L[kLsMaxR][kLsMaxR];   // L[j][k] = <v_k, v_j>, j < k
    V H[kLsMaxR][kLsMaxR];   // H[i][k]: column i of the rotated Hessenberg matrix
    V cs[kLsMaxR], sn[kLsMaxR], s[kLsMaxR + 1], y[kLsMaxR], scl[kLsMaxR + 1];
    V tot[kLsVals];          // sums of the last reduction
    V coef[kLsMaxR];         // h_k scl_k
    V aw[kLsMaxR];           // <w, v_k>
    V hp[4][kLsMaxR];        // parts of L a
    V rc[kLsMaxR], rs[kLsMaxR], rt[kLsMaxR];
    V pd[kLsWarps * 8];      // dots of one warp each
    V pw[kLsWarps];          // |w|^2 of one warp each
    V grp[kLsThreads];       // partial sums of the reduction
    V hlast;                 // last entry of the rotated column before the new rotation
    double resid, normb, beta;
    int flag;
    int lmax;                // largest |L_kj| of the cycle (bits of a float)
    int Ew;                  // exponent of the last |w| before its projection
};

__device__ __forceinline__ float ls_add(const float (&p)[16]) {
    float a = p[0];
#pragma unroll
    for (int u = 1; u < 16; ++u) a += p[u];
    return a;
}
__device__ __forceinline__ double ls_add(const double (&p)[16]) { return fx_sum(p); }
__device__ __forceinline__ float ls_sum8(const float (&v)[8], int lane) { return warp_sum8(v, lane); }
__device__ __forceinline__ double ls_sum8(const double (&v)[8], int lane) { return warp_fx_sum8(v, lane); }

__device__ __forceinline__ float ls_sum1(float v) { return warp_sum(v); }
__device__ __forceinline__ double ls_sum1(double v) {
    const double one[1] = {v};
    return warp_fx_sum(one);
}

__device__ __forceinline__ float ls_rsqrt(float x) { return 1.0f / sqrtf(x); }
__device__ __forceinline__ double ls_rsqrt(double x) { return rsqrt_fp64(x); }

// The n block partials in part[block][value] summed over the blocks into tot
// (all blocks the same bits): thread t takes value t % n over every G-th
// block, 16 loads in flight, then the G sums are added.  Consecutive threads
// read consecutive values of a block.
template <class V>
__device__ void ls_sum_parts(const V* part, int n, V* grp, V* tot) {
    const int G = min(kLsThreads / n, 16);
    const int gq = (int)threadIdx.x / n, k = (int)threadIdx.x - gq * n;
    const int nb = (int)gridDim.x;
    if (gq < G) {
        V acc = V(0);
        for (int b0 = gq; b0 < nb; b0 += 16 * G) {
            V p[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                const int b = b0 + u * G;
                p[u] = b < nb ? __ldcg(part + (size_t)b * kLsVals + k) : V(0);
            }
            const V s = ls_add(p);
            acc = b0 == gq ? s : acc + s;
        }
        grp[threadIdx.x] = acc;
    }
    __syncthreads();
    if ((int)threadIdx.x < n) {
        V p[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) p[u] = u < G ? grp[u * n + threadIdx.x] : V(0);
        tot[threadIdx.x] = ls_add(p);
    }
    __syncthreads();
}

// SMEM: the block's parts of w and v_i lie in shared memory (a pointer to either would make every access generic)
template <class V, bool SMEM>
__global__ void __launch_bounds__(kLsThreads, 1) k_gmres_ls(GmLsArgs<V> a) {
    constexpr bool kMixed = sizeof(V) == 4;
    extern __shared__ __align__(16) unsigned char ls_dyn[];
    LsSmall<V>& q = *reinterpret_cast<LsSmall<V>*>(ls_dyn);
    V* const sbuf = reinterpret_cast<V*>(ls_dyn + ((sizeof(LsSmall<V>) + 15) & ~(size_t)15));
    __shared__ BalShared<kLsWarps, V> bsh;
    __shared__ BalShared<kLsWarps, double> bshd;
    __shared__ int st_sh;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t s0 = (int64_t)blockIdx.x * a.nslices / gridDim.x;
    const int64_t s1 = (int64_t)(blockIdx.x + 1) * a.nslices / gridDim.x;
    const int64_t base = s0 * 32;
    const int nl = (int)(s1 - s0) * 32;
    const int R = a.R;
    unsigned long long epoch = 0;
    int it = 0, cycles = 0;  // Arnoldi steps, cycles
    // a run of at most kBalMaxSlices slices plans its column split once
    const bool planned = s1 - s0 <= kBalMaxSlices;
    __shared__ WalkRange wrs[kLsWarps];
    if (planned) {
        sell_block_plan<kLsWarps, V>(bsh, a.ptr, s0, (int)(s1 - s0));
        if (lane == 0) wrs[warp] = sell_block_range(bsh, (int)(s1 - s0));
        __syncwarp();
    }
    // the head of the block's part of B in shared memory: its slices [0, cs)
    int cs = 0;
    V* const cval = sbuf + 2 * a.nloc;
    int32_t* const ccol = reinterpret_cast<int32_t*>(cval + a.ccap);
    if (SMEM && planned) {
        const int S = (int)(s1 - s0);
        while (cs < S && 32 * bsh.P[cs + 1] <= a.ccap) ++cs;
        const int32_t pb = __ldg(a.ptr + s0);
        for (int k = threadIdx.x; k < 32 * bsh.P[cs]; k += kLsThreads) {
            cval[k] = __ldg(a.bval + pb + k);
            ccol[k] = __ldg(a.cols + pb + k);
        }
    }

    // one reduction: the block's n partials are in part[epoch & 1][block]
    auto reduce = [&](int n) -> bool {
        const V* part = a.part + (size_t)(epoch & 1) * gridDim.x * kLsVals;
        if (!ar_arrive_wait(a.g, epoch, &st_sh)) return false;
        ++epoch;
        ls_sum_parts<V>(part, n, q.grp, q.tot);
        return true;
    };

    PkState pkn;
    unsigned pepoch = 0;
    unsigned long long plast[2] = {0ull, 0ull}, plast2[2] = {0ull, 0ull};
    if (threadIdx.x == 0) {
        q.Ew = kPkUnknown;
    }
    bool first = true;
    for (;;) {
        // ---- residual r = b - A x (FP64) into basis_0, its norm ----
        {
            double v[2] = {0., 0.};
            const double* x = a.x;
            V* const V0 = a.basis + base;
            for (int64_t c0 = s0; c0 < s1; c0 += kBalMaxSlices)
                sell_block_balanced<kLsWarps, double>(
                    bshd, a.ptr, a.col, a.aval, c0, (int)(s1 - c0 < kBalMaxSlices ? s1 - c0 : kBalMaxSlices),
                    [&](int32_t j) { return kld(x + j); },
                    [&](int64_t s, double ax) {
                        const int32_t row = __ldg(a.perm + s * 32 + lane);
                        double r = 0., bi = 0.;
                        if (row >= 0) {
                            bi = a.b[row];
                            r = bi - ax;
                            if (a.left) {
                                r = r / a.diag[row];
                                bi = bi / a.diag[row];
                            }
                        }
                        V0[(s - s0) * 32 + lane] = (V)r;
                        if (SMEM) sbuf[(s - s0) * 32 + lane] = (V)r;
                        v[0] += r * r;
                        if (first) v[1] += bi * bi;
                    });
            double o[2];
            if (!grid_allreduce<double, 2>(a.g, epoch, v, o)) return;
            if (threadIdx.x == 0) {
                if (first) {
                    const double nb = sqrt(o[1]);
                    q.normb = nb == 0.0 || !a.rel ? 1.0 : nb;
                }
                q.beta = sqrt(o[0]);
                q.resid = q.beta / q.normb;
                q.scl[0] = (V)(1.0 / q.beta);
                q.s[0] = (V)q.beta;
                q.lmax = 0;
            }
            __syncthreads();
            first = false;
        }
        const double inv_normb = 1.0 / q.normb;
        const double inner_stop = fmax(a.inner_floor * q.beta, 0.5 * a.tol * q.normb);  // mixed: end of a cycle
        double resid = q.resid;
        if (resid <= a.tol || it >= a.max_iter) {
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                // the reference counts a cycle that ends on the new residual one further; the mixed solver
                // counts Arnoldi steps
                *a.out_iter = resid <= a.tol ? (kMixed || it == 0 ? it : it + 1) : -1 - it;
                *a.out_resid = resid;
                *a.out_cycles = cycles;
            }
            return;
        }
        ++cycles;
        // ---- Arnoldi steps ----
        const int steps = kMixed ? R : R - 1;
        bool done = false;
        int i = 0;
        V* ws = SMEM ? sbuf + a.nloc : nullptr;  // this block's part of w, then of the next v_i
        V* vs = SMEM ? sbuf : nullptr;           // of v_i
        while (i < steps && it < a.max_iter) {
            const V* const Vi = a.basis + (size_t)i * a.ld;
            V* const W = a.basis + (size_t)(i + 1) * a.ld;
            const V sci = q.scl[i];
            V* const wl = SMEM ? ws : W + base;
            const V* const vl = SMEM ? vs : Vi + base;
            for (int64_t c0 = s0; c0 < s1; c0 += kBalMaxSlices) {
                const int S = (int)(s1 - c0 < kBalMaxSlices ? s1 - c0 : kBalMaxSlices);
                if (!planned) {
                    sell_block_plan<kLsWarps, V>(bsh, a.ptr, c0, S);
                    if (lane == 0) wrs[warp] = sell_block_range(bsh, S);
                    __syncwarp();
                }
                sell_block_walk_range(
                    bsh, c0, S, wrs[warp],
                    [&](int64_t s, int32_t k, int32_t n) {
                        auto gather = [&](int32_t j) { return kld(Vi + j); };
                        if (SMEM && s - s0 < cs) {
                            const int e = 32 * (bsh.P[s - s0] + k) + lane;
                            return sell_row_walk<true, V>(ccol + e, cval + e, n, gather);
                        }
                        return sell_row_range<V>(a.ptr, a.cols, a.bval, s, lane, k, n, gather);
                    },
                    [&](int64_t s, V acc) { wl[(s - s0) * 32 + lane] = sci * acc; });
            }
            // Dots of w and v_i with the basis: a warp takes four basis vectors and, while there are
            // fewer than kLsWarps such groups, every parts-th 32 rows of the block.
            {
                const int groups = (i + 4) >> 2, parts = kLsWarps / groups;
                const int grp = warp % groups, pt = warp / groups;
                if (pt < parts) {
                    V d[8], dw = V(0);
#pragma unroll
                    for (int u = 0; u < 8; ++u) d[u] = V(0);
                    const V* vk[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) vk[u] = a.basis + (size_t)min(4 * grp + u, i) * a.ld + base;
                    const int nk = i + 1 - 4 * grp;
#pragma unroll 2
                    for (int e = pt * 32 + lane; e < nl; e += 32 * parts) {
                        const V we = wl[e], ve = vl[e];
                        if (grp == 0) dw += we * we;
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (u < nk) {
                                const V t = kld(vk[u] + e);
                                d[u] += we * t;
                                d[4 + u] += ve * t;
                            }
                    }
                    const V tot = ls_sum8(d, lane);
                    if ((lane & 3) == 0) q.pd[warp * 8 + warp_sum8_index(lane)] = tot;
                    if (grp == 0) {
                        const V t = ls_sum1(dw);
                        if (lane == 0) q.pw[pt] = t;
                    }
                }
                __syncthreads();
                // thread j: <w, v_j> (j <= i), <v_i, v_k> (i of them), then |w|^2, over the block; a packed
                // reduction, the unit of each from |w| of the step before (1 for <v_i, v_k>)
                const int n = 2 * i + 2, j = threadIdx.x;
                V sum = V(0);
                if (j < n - 1) {
                    const int u = j <= i ? 0 : 4, k = j <= i ? j : j - i - 1;
                    const V* p = q.pd + (k >> 2) * 8 + u + (k & 3);
                    sum = p[0];
                    for (int t = 1; t < parts; ++t) sum += p[t * groups * 8];
                    sum *= q.scl[k];
                    if (j > i) sum *= sci;
                } else if (j == n - 1) {
                    sum = q.pw[0];
                    for (int t = 1; t < parts; ++t) sum += q.pw[t];
                }
                int st = 1;
                const int Ew = q.Ew;
                if (Ew != kPkUnknown) {
                    st = 0;
                    if (j < n) {
                        const int E = j <= i ? Ew : j < n - 1 ? 0 : 2 * Ew + 1;
                        V val;
                        if constexpr (kMixed) {
                            bool bad;
                            const long long t = pk_fix(sum, E, &bad);
                            unsigned long long diff = 0;
                            st = pk_exchange(a.pkd, pepoch, plast, j, t, !bad, &diff);
                            val = pk_value(pk_sum(diff), E);
                        } else {
                            bool bad;
                            long long hi, lo;
                            pk_fix(sum, E, &hi, &lo, &bad);
                            const bool fits = pk_carry(&hi, &lo) && !bad;
                            unsigned long long* w = a.pkd.w + (pepoch & 1) * kPkWords + 2 * j;
                            red_relaxed_add_u64(w + 1, pk_word(lo, !fits));  // both words on their way before the waits
                            unsigned long long dh = 0, dl = 0;
                            st = pk_exchange(a.pkd, pepoch, plast, 2 * j, hi, fits, &dh);
                            if (!pk_wait(w + 1, pepoch & 1 ? plast2[1] : plast2[0], a.pkd.status, &dl)) st = 2;
                            val = pk_value(pk_sum(dh), (long long)(dl >> 16), E);
                        }
                        q.tot[j] = val;
                        // |w| far below the unit's: the dots would lack bits
                        if (j == n - 1 && pk_exp(val) < E - 2 * (kMixed ? kPkDrop32 : kPkDrop64)) st = max(st, 1);
                    }
                    ++pepoch;
                    if (__syncthreads_or(st == 2)) return;
                    st = __syncthreads_or(st);
                }
                if (st) {  // no |w| yet, or a value outside the range of its unit
                    if (j < n) a.part[((size_t)(epoch & 1) * gridDim.x + blockIdx.x) * kLsVals + j] = sum;
                    if (!reduce(n)) return;
                }
            }
            // h = (I + L)^{-1} a.  While max |L|^2 is below the rounding of a, h = a - L a to that rounding: a
            // product over four warps; else forward substitution, two entries per lane of warp 0.
            if ((int)threadIdx.x <= i) {
                const int k = threadIdx.x;
                q.aw[k] = q.tot[k];
                if (k < i) {
                    const V l = q.tot[i + 1 + k];
                    q.L[k][i] = l;
                    atomicMax(&q.lmax, __float_as_int(fabsf((float)l)));
                }
            }
            __syncthreads();
            const float lm = __int_as_float(q.lmax);
            if (lm * lm * (float)(i + 1) <= (kMixed ? 1.4e-8f : 2.7e-17f)) {
                if (warp < 4)
                    for (int k = lane; k <= i; k += 32) {
                        V t = V(0);
                        for (int j = warp; j < k; j += 4) t += q.L[j][k] * q.aw[j];
                        q.hp[warp][k] = t;
                    }
                __syncthreads();
                if ((int)threadIdx.x <= i) {
                    const int k = threadIdx.x;
                    const V h = q.aw[k] - ((q.hp[0][k] + q.hp[1][k]) + (q.hp[2][k] + q.hp[3][k]));
                    q.H[i][k] = h;
                    q.coef[k] = h * q.scl[k];
                }
            } else if (warp == 0) {
                V h0 = lane <= i ? q.aw[lane] : V(0);
                V h1 = lane + 32 <= i ? q.aw[lane + 32] : V(0);
                for (int j = 0; j < i; ++j) {
                    const V hj = __shfl_sync(0xffffffffu, j < 32 ? h0 : h1, j & 31);
                    if (lane > j && lane <= i) h0 -= q.L[j][lane] * hj;
                    if (lane + 32 > j && lane + 32 <= i) h1 -= q.L[j][lane + 32] * hj;
                }
                if (lane <= i) {
                    q.H[i][lane] = h0;
                    q.coef[lane] = h0 * q.scl[lane];
                }
                if (lane + 32 <= i) {
                    q.H[i][lane + 32] = h1;
                    q.coef[lane + 32] = h1 * q.scl[lane + 32];
                }
            }
            __syncthreads();
            // the last warp applies the previous rotations to the new column while the others update w
            if (warp == kLsWarps - 1) {
                V* const hc = q.H[i];
                for (int k = lane; k < i; k += 32) {
                    const V hk = hc[k + 1];
                    q.rc[k] = q.cs[k] * hk;
                    q.rs[k] = q.sn[k] * hk;
                }
                __syncwarp();
                if (lane == 0) {
                    V t = hc[0];
                    for (int k = 0; k < i; ++k) {
                        q.rt[k] = t;
                        t = q.rc[k] - q.sn[k] * t;
                    }
                    q.hlast = t;
                }
                __syncwarp();
                for (int k = lane; k < i; k += 32) hc[k] = q.cs[k] * q.rt[k] + q.rs[k];
            }
            // w -= V h on the block's rows, |w|^2
            V nrm[1] = {V(0)};
            for (int e = threadIdx.x; e < nl; e += kLsThreads) {
                V acc[4] = {wl[e], V(0), V(0), V(0)};
                const V* vk = a.basis + base + e;
                int k = 0;
                for (; k + 7 <= i; k += 8) {
                    V t[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) t[u] = kld(vk + (size_t)(k + u) * a.ld);
#pragma unroll
                    for (int u = 0; u < 8; ++u) acc[u & 3] -= q.coef[k + u] * t[u];
                }
                for (; k <= i; ++k) acc[k & 3] -= q.coef[k] * kld(vk + (size_t)k * a.ld);
                const V w = (acc[0] + acc[1]) + (acc[2] + acc[3]);
                W[base + e] = w;
                if (SMEM) ws[e] = w;
                nrm[0] += w * w;
            }
            V o[1];
            if (!packed_allreduce<1>(a.pkn, pkn, a.g, epoch, nrm, o, true)) return;
            ++it;
            if (warp == 0) {
                // lane 0: 1 / |w|; lane 1: 1 / r, r = |(hlast, |w|)|
                const V t = q.hlast, n2 = o[0];
                const V arg = lane == 1 ? t * t + n2 : n2;
                const V inv = arg > V(0) ? ls_rsqrt(arg) : V(0);
                const V ih = __shfl_sync(0xffffffffu, inv, 0), ir = __shfl_sync(0xffffffffu, inv, 1);
                if (lane == 0) {
                    const V hn = n2 * ih;  // 0 (or NaN) where |w|^2 is
                    const bool zero = n2 == V(0);
                    const V c = zero ? V(1) : t * ir, s = zero ? V(0) : hn * ir;
                    q.scl[i + 1] = ih;
                    const int e2 = pk_exp(q.tot[2 * i + 1]);
                    q.Ew = e2 == kPkUnknown ? kPkUnknown : e2 >> 1;
                    q.cs[i] = c;
                    q.sn[i] = s;
                    q.H[i][i] = c * t + s * hn;
                    const V si = q.s[i];
                    q.s[i] = c * si;
                    q.s[i + 1] = -s * si;
                    const double est = fabs((double)q.s[i + 1]);
                    if (kMixed) {
                        q.flag = est <= inner_stop || zero;
                    } else {
                        q.resid = est * inv_normb;
                        q.flag = q.resid <= a.tol;
                    }
                }
            }
            __syncthreads();
            resid = q.resid;
            done = q.flag != 0;
            ++i;
            if (SMEM) {
                V* t = ws;
                ws = vs;
                vs = t;
            }
            if (done) break;
        }
        // ---- y = H^{-1} s on the leading i x i triangle, x += P^{-1} V y ----
        const int kk = i - 1;
        if (warp == 0) {
            V y0 = lane <= kk ? q.s[lane] : V(0), y1 = lane + 32 <= kk ? q.s[lane + 32] : V(0);
            const V d0 = lane <= kk ? V(1) / q.H[lane][lane] : V(0);
            const V d1 = lane + 32 <= kk ? V(1) / q.H[lane + 32][lane + 32] : V(0);
            for (int j = kk; j >= 0; --j) {
                V yj = j < 32 ? y0 * d0 : y1 * d1;
                yj = __shfl_sync(0xffffffffu, yj, j & 31);
                if (lane < j) y0 -= q.H[j][lane] * yj;
                if (lane + 32 < j) y1 -= q.H[j][lane + 32] * yj;
            }
            if (lane <= kk) q.coef[lane] = y0 * d0 * q.scl[lane];
            if (lane + 32 <= kk) q.coef[lane + 32] = y1 * d1 * q.scl[lane + 32];
        }
        __syncthreads();
        for (int e = threadIdx.x; e < nl; e += kLsThreads) {
            const int32_t row = __ldg(a.perm + base + e);
            if (row < 0) continue;
            V z = V(0);
            const V* vk = a.basis + base + e;
            for (int k = 0; k <= kk; ++k) z += q.coef[k] * kld(vk + (size_t)k * a.ld);
            if (a.binv) a.zrow[row] = z;
            else a.x[row] += a.left ? (double)z : (double)z / a.diag[row];
        }
        if (!kMixed && done) {  // converged on the rotated residual
            if (a.binv && !grid_sync_ar(a.g, epoch)) return;
        } else if (!grid_sync_ar(a.g, epoch)) {
            return;
        }
        if (a.binv) {
            const int64_t half = a.m / 2;
            for (int64_t e = blockIdx.x * (int64_t)kLsThreads + threadIdx.x; e < half; e += (int64_t)gridDim.x * kLsThreads) {
                const double za = (double)kld(a.zrow + e), zb = (double)kld(a.zrow + e + half);
                const double* q4 = a.binv + 4 * e;
                a.x[e] += q4[0] * za + q4[1] * zb;
                a.x[e + half] += q4[2] * za + q4[3] * zb;
            }
            if ((kMixed || !done) && !grid_sync_ar(a.g, epoch)) return;
        }
        if (!kMixed && done) {
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                *a.out_iter = it;
                *a.out_resid = resid;
                *a.out_cycles = cycles;
            }
            return;
        }
    }
}

// the SELL columns as slots (pad entries: the slot of their row, or 0)
__global__ void k_ls_cols(int64_t npad, const int32_t* __restrict__ col, const int32_t* __restrict__ iperm,
                          int32_t* __restrict__ cols) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < npad; i += (int64_t)gridDim.x * blockDim.x)
        cols[i] = iperm[col[i]];
}

// once per pattern of the matrix in handle id
int ensure_slot_cols(Context* c, CSR& A, int id, const int32_t** cols) {
    Sell& S = A.sell;
    TF_TRY(ensure(c, c->sell_cols[id], (size_t)(S.npad > 0 ? S.npad : 1)));
    if (c->sell_cols_gen[id] != S.pattern_gen) {
        TF_TRY(ensure_sell_iperm(c, A));
        k_ls_cols<<<grid_for(c, S.npad), kBlock, 0, c->stream>>>(S.npad, S.col, S.iperm, c->sell_cols[id].p);
        ++c->launches;
        TF_CUDA(c, cudaGetLastError());
        c->sell_cols_gen[id] = S.pattern_gen;
    }
    *cols = c->sell_cols[id].p;
    return TF_OK;
}

}  // namespace

// Modified Gram-Schmidt GMRES on this kernel.  V = double: method 0 (right) or
// 1 (left, point Jacobi only); V = float: the mixed-precision solver (right).
template <class V>
int gmres_ls(Context* c, CSR& A, const double* b, double* x, int R, int left, int* max_iter, double* tol, int rel) {
    const int id = (int)(&A - c->mats);
    const int64_t m = A.m;
    const bool block = id == TF_MAT_BLOCK;
    TF_TRY(ensure_diag(c, A));
    TF_TRY(ensure_sell(c, A, false));
    const int32_t* cols = nullptr;
    TF_TRY(ensure_slot_cols(c, A, id, &cols));
    const V* bval = nullptr;
    TF_TRY(gmres_operator<V>(c, A, left, &bval));
    TimedLaunch tl(c, TF_K_GMRES);
    const int64_t ns = A.sell.used, ld = ns * 32;
    // at least two slices per block: a block's share of the reductions (its
    // partials are read by every other block) outweighs less work per block
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(std::min(c->num_sms, kPkMaxBlocks), ns / 2));
    DBuf<V>& basis = *reinterpret_cast<DBuf<V>*>(sizeof(V) == 4 ? (void*)&c->gm2_v32 : (void*)&c->gm2_v64);
    TF_TRY(ensure(c, basis, (size_t)(R + 1) * ld + (block ? (size_t)m : 0)));
    const size_t part_v = (size_t)2 * blocks * kLsVals, part_r = (size_t)2 * blocks * kArMax;
    TF_TRY(ensure(c, c->kry_part, part_v + 2 * part_r + 16));
    TF_TRY(ensure(c, c->kry_bar, 4));
    TF_TRY(ensure(c, c->kry_iters, 4));
    TF_TRY(ensure(c, c->kry_resid, 1));
    TF_CUDA(c, cudaMemsetAsync(c->kry_bar.p, 0, 4 * sizeof(unsigned), c->stream));
    TF_CUDA(c, cudaMemsetAsync(c->status.p, 0, 4 * sizeof(int), c->stream));
    unsigned long long* pw = nullptr;
    TF_TRY(packed_words(c, 2, &pw));
    int64_t room = 0;
    TF_TRY(max_dynamic_smem(c, (const void*)k_gmres_ls<V, true>, &room));
    const size_t small = (sizeof(LsSmall<V>) + 15) & ~(size_t)15;
    const int64_t run = 32 * ((ns + blocks - 1) / blocks);  // slots of the largest run
    const int64_t both = (int64_t)small + 2 * run * (int64_t)sizeof(V);
    const bool smem = both <= room;  // else w and v_i are read from the basis
    // what is left keeps the head of every block's part of B (at most the largest run, guessed at 9/8 of the mean)
    const int64_t mean = A.sell.npad / blocks;
    int64_t ccap = smem ? std::min((room - both) / (int64_t)(sizeof(V) + 4), mean + mean / 8 + 1024) & ~(int64_t)31 : 0;
    if (ccap < 0) ccap = 0;
    const size_t dyn = smem ? (size_t)(both + ccap * (int64_t)(sizeof(V) + 4)) : small;
    const void* fn = smem ? (const void*)k_gmres_ls<V, true> : (const void*)k_gmres_ls<V, false>;
    if (!smem) TF_TRY(max_dynamic_smem(c, fn, &room));
    int per_sm = 0;
    TF_CUDA(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kLsThreads, dyn));
    if (per_sm < 1) return set_err(c, TF_ERR_CUDA, "gmres: kernel does not fit the SM");
    GmLsArgs<V> g{};
    g.nslices = ns;
    g.m = m;
    g.perm = A.sell.perm;
    g.ptr = A.sell.ptr;
    g.col = A.sell.col;
    g.cols = cols;
    g.bval = bval;
    g.aval = A.sell.v64;
    g.b = b;
    g.x = x;
    g.diag = block ? nullptr : A.diag;
    g.binv = block ? c->gm2_binv.p : nullptr;
    g.basis = basis.p;
    g.ld = ld;
    g.zrow = block ? basis.p + (size_t)(R + 1) * ld : nullptr;
    g.part = reinterpret_cast<V*>(c->kry_part.p);
    g.g.count = reinterpret_cast<unsigned long long*>(c->kry_bar.p);
    g.g.partd = c->kry_part.p + part_v;
    g.g.partf = reinterpret_cast<float*>(c->kry_part.p + part_v + part_r);
    g.g.status = c->status.p;
    g.pkd = PackedAR{pw, c->status.p};
    g.pkn = PackedAR{pw + 2 * kPkWords, c->status.p};
    g.R = R;
    g.max_iter = *max_iter;
    g.rel = rel;
    g.left = left;
    g.nloc = smem ? (int)run : 0;
    g.ccap = (int)ccap;
    g.tol = *tol;
    g.inner_floor = 1e-5;
    g.out_iter = c->kry_iters.p;
    g.out_cycles = c->kry_iters.p + 1;
    g.out_resid = c->kry_resid.p;
    void* args[] = {&g};
    TF_CUDA(c, cudaLaunchCooperativeKernel(fn, blocks, kLsThreads, args, dyn, c->stream));
    ++c->launches;
    int it[2] = {0, 0};
    double res = 0.;
    TF_CUDA(c, cudaMemcpyAsync(it, c->kry_iters.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    TF_CUDA(c, cudaMemcpyAsync(&res, c->kry_resid.p, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    int st = 0;
    TF_TRY(sync_status(c, &st));
    if (st) return set_err(c, st, "gmres: grid barrier watchdog fired");
    c->last_refinements = it[1];
    *tol = res;
    *max_iter = it[0] >= 0 ? it[0] : -1 - it[0];
    return it[0] >= 0 ? TF_OK
                      : set_err(c, TF_ERR_NOT_CONVERGED, sizeof(V) == 4 ? "gmres (mixed): no convergence within max_iter"
                                                                        : "gmres: no convergence within max_iter");
}

template int gmres_ls<double>(Context*, CSR&, const double*, double*, int, int, int*, double*, int);
template int gmres_ls<float>(Context*, CSR&, const double*, double*, int, int, int*, double*, int);

}  // namespace tf

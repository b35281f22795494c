// Cut classification and interface DOF numbering.
//
// IdxDescCL::DistributeDOFs (misc/problem.cpp:283-336) walks the tets in
// triangulation order and gives every vertex (and, for P2, edge) of an active
// tet the next number on first touch.  Here that serial walk becomes three
// data-parallel steps with the same result:
//   1. classify: distance() of every tet on its 10 level-set values
//      (geom/subtriangulation.tpp:38-46), on a brick one thread per cube, which
//      reads the cube's 27 nodes once for its six tets; activity bits and a
//      count per tile, then the active tets are written in tet order;
//   2. first touch: each active tet r offers the key r*nloc + slot to each of
//      its vertices/edges with atomicMin -- the minimum key is exactly the
//      position of the first touch in the reference's walk;
//   3. ranking: the keys are unique, so a scan over the key space turns every
//      owned key into its DOF number.
#include <climits>
#include <cstring>

#include "tf_internal.cuh"

namespace tf {

__device__ inline void set_status(int* st, int code, int64_t where) {
    if (atomicCAS(st, 0, code) == 0) st[1] = (int)where;
}

// The distance test on the IEEE-754 bit patterns, with integer operations
// only: GB300 issues FP64 compares on its narrow FP64 pipe, and ten values per
// tet made classification FP64-bound.  For a double with bits b and
// magnitude bits m = b & 0x7ff..f: sign(d) (misc/utils.h:810-813) is 0 for
// m == 0 (+-0) and for NaN (m > 0x7ff0..0, where both comparisons of sign()
// are false), else -1 or +1 by the sign bit; for non-NaN values |a| < |c| iff
// m_a < m_c, so min |f| is the minimum of the m.
struct DistTest {
    unsigned long long dmag;  // magnitude bits of dist (when dist >= 0)
    int dmag_ok;              // dist >= 0: min |f| <= dist is dmag compare
    int mixed_active;         // 0 <= dist: a tet with a sign change is active
};

// A group of tets (the six of a cube of a brick, or one tet of an uploaded
// mesh) has one byte of activity bits; a tile is kTile groups of one block.
constexpr int kTileThreads = 256;
constexpr int kTilePer = 2;
constexpr int kTile = kTileThreads * kTilePer;

// The 27 nodes of a cube: vertices 0..7 at (d3 d2 d1), then the edges of the
// seven direction classes (001, 010, 100, 011, 101, 110, 111) by the offset of
// their lower vertex; node masks of the six tets.
struct CubeMasks {
    unsigned tet[6];
};
static CubeMasks cube_masks() {
    CubeMasks C;
    static const int base[7] = {8, 12, 16, 20, 22, 24, 26};
    for (int l = 0; l < 6; ++l) {
        unsigned m = 0;
        int p[4][3];
        for (int k = 0; k < 4; ++k) {
            kuhn_offset(l, k, p[k][0], p[k][1], p[k][2]);
            m |= 1u << (p[k][0] * 4 + p[k][1] * 2 + p[k][2]);
        }
        for (int k = 0; k < 6; ++k) {
            const int *a = p[ev0(k)], *b = p[ev1(k)];
            const int d3 = b[0] - a[0], d2 = b[1] - a[1], d1 = b[2] - a[2];
            // the lower vertex's offset along the directions the edge does not take
            int sub = 0;
            if (!d3) sub = a[0];
            if (!d2) sub = 2 * sub + a[1];
            if (!d1) sub = 2 * sub + a[2];
            m |= 1u << (base[edir_class(d3, d2, d1)] + sub);
        }
        C.tet[l] = m;
    }
    return C;
}

struct NodeBits {
    unsigned pos = 0, neg = 0, zero = 0, near = 0;  // sign, exact zero, |f| <= dist
};
__device__ __forceinline__ void node_bit(NodeBits& B, int bit, long long f, const DistTest& D) {
    const unsigned long long m = (unsigned long long)f & 0x7fffffffffffffffull;
    const bool zero = m == 0ull, nan = m > 0x7ff0000000000000ull;
    B.pos |= (!zero && !nan && f > 0 ? 1u : 0u) << bit;
    B.neg |= (!zero && !nan && f < 0 ? 1u : 0u) << bit;
    B.zero |= (zero ? 1u : 0u) << bit;
    B.near |= (D.dmag_ok && m <= D.dmag ? 1u : 0u) << bit;
}
// activity of the tet with nodes `mask` (10 of them), *z set for an exact zero on a cut tet
__device__ __forceinline__ bool tet_active(const NodeBits& B, unsigned mask, const DistTest& D, bool* z) {
    if ((B.pos & mask) == mask || (B.neg & mask) == mask) return (B.near & mask) != 0;  // distance() = min |f|
    *z = (B.zero & mask) != 0;
    return D.mixed_active;  // distance() = 0
}

// f(bit, index, edge) for the 27 nodes of cube (i1, i2, i3): offsets v0, e0 into the vertices and edges
template <class F>
__device__ __forceinline__ void cube_nodes(const Brick& B, int i1, int i2, int i3, int64_t v0, int64_t e0, F f) {
    const int n1 = B.n1, n2 = B.n2;
#pragma unroll
    for (int k = 0; k < 8; ++k)
        f(k, v0 + ((int64_t)(i3 + (k >> 2)) * (n2 + 1) + i2 + (k >> 1 & 1)) * (n1 + 1) + i1 + (k & 1), false);
    int bit = 8;
#pragma unroll
    for (int cls = 0; cls < 7; ++cls) {
        constexpr int code[7] = {1, 2, 4, 3, 5, 6, 7};
        const int d3 = code[cls] >> 2 & 1, d2 = code[cls] >> 1 & 1, d1 = code[cls] & 1;
        const int64_t off = e0 + B.eoff[cls];
#pragma unroll
        for (int a3 = 0; a3 < 2 - d3; ++a3)
#pragma unroll
            for (int a2 = 0; a2 < 2 - d2; ++a2)
#pragma unroll
                for (int a1 = 0; a1 < 2 - d1; ++a1)
                    f(bit++, off + ((int64_t)(i3 + a3) * (n2 + 1 - d2) + i2 + a2) * (n1 + 1 - d1) + i1 + a1, true);
    }
}

// Bound: instruction issue, then the level set read once (8 B per node; 27 loads
// per six tets, where a thread per tet took 60 and wrote a 4-byte flag that the
// scan and the compaction read and rewrote).  A node's high word tells its sign
// unless its exponent is 0 or all ones (zero, subnormal, infinity, NaN); cubes
// with such a node, and every cube when dist > 0, test all bits.
// Classification to compacted list on GB300: 256 ellipsoids (141.5M tets, 1.5 GB
// of values) 4.49 -> 0.74 ms, P1 128^3 (12.6M tets) 0.36 -> 0.07 ms.
template <bool BRICK>
__global__ void __launch_bounds__(kTileThreads) k_classify(MeshView M, int64_t ngroups, const double* __restrict__ lsv,
                                                           const double* __restrict__ lse, DistTest D, CubeMasks C,
                                                           uint8_t* __restrict__ bits, int32_t* __restrict__ tile_cnt,
                                                           int* __restrict__ status) {
    const long long* bv = reinterpret_cast<const long long*>(lsv);
    const long long* be = reinterpret_cast<const long long*>(lse);
    __shared__ int inst0, wsum[kTileThreads / 32];
    const int64_t first = (int64_t)blockIdx.x * kTile;
    if (BRICK && M.nbatch) {
        if (threadIdx.x == 0) inst0 = batch_find(M.tstart, M.nbatch, 6 * first);
        __syncthreads();
    }
    int inst = BRICK && M.nbatch ? inst0 : 0;
    const bool band = D.dmag_ok && D.dmag != 0;  // tets without a sign change can be active
    int cnt = 0;
    for (int j = 0; j < kTilePer; ++j) {
        const int64_t g = first + j * kTileThreads + threadIdx.x;
        if (g >= ngroups) break;
        NodeBits B;
        unsigned act = 0;
        if constexpr (BRICK) {
            int64_t v0 = 0, e0 = 0;
            uint32_t cube = (uint32_t)g;
            const Brick* bp = &M.b;
            if (M.nbatch) {
                while (inst + 1 < M.nbatch && 6 * g >= M.tstart[inst + 1]) ++inst;
                const BatchBrick& I = M.batch[inst];
                bp = &I.b;
                v0 = I.v0;
                e0 = I.e0;
                cube = (uint32_t)(g - I.t0 / 6);
            }
            const uint32_t r = cube / (uint32_t)bp->n1;
            const int i1 = (int)(cube - r * bp->n1);
            const int i3 = (int)(r / (uint32_t)bp->n2), i2 = (int)(r - (uint32_t)i3 * bp->n2);
            unsigned odd = band ? 1u : 0u;
            if (!band) {
                unsigned neg = 0;
                cube_nodes(*bp, i1, i2, i3, v0, e0, [&](int bit, int64_t i, bool edge) {
                    const int h = __ldg(reinterpret_cast<const int*>(edge ? be : bv) + 2 * i + 1);
                    neg |= (unsigned)h >> 31 << bit;
                    odd |= ((unsigned)h & 0x7ff00000u) - 0x100000u >= 0x7fe00000u;
                });
#pragma unroll
                for (int l = 0; l < 6; ++l) {
                    const unsigned s = neg & C.tet[l];
                    act |= (s != 0 && s != C.tet[l] && D.mixed_active ? 1u : 0u) << l;
                }
            }
            if (odd) {
                act = 0;
                cube_nodes(*bp, i1, i2, i3, v0, e0,
                           [&](int bit, int64_t i, bool edge) { node_bit(B, bit, __ldg((edge ? be : bv) + i), D); });
#pragma unroll
                for (int l = 0; l < 6; ++l) {
                    bool z = false;
                    act |= (tet_active(B, C.tet[l], D, &z) ? 1u : 0u) << l;
                    if (z) set_status(status, TF_ERR_ZERO_NODE, 6 * g + l);
                }
            }
        } else {
            int32_t v[4], e[6];
            mesh_tet(M, g, v, e);
#pragma unroll
            for (int k = 0; k < 4; ++k) node_bit(B, k, __ldg(bv + v[k]), D);
#pragma unroll
            for (int k = 0; k < 6; ++k) node_bit(B, 4 + k, __ldg(be + e[k]), D);
            bool z = false;
            act = tet_active(B, 0x3ffu, D, &z) ? 1u : 0u;
            if (z) set_status(status, TF_ERR_ZERO_NODE, g);
        }
        bits[g] = (uint8_t)act;
        cnt += __popc(act);
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0;
        for (int w = 0; w < kTileThreads / 32; ++w) s += wsum[w];
        tile_cnt[blockIdx.x] = s;
    }
}

// exclusive offsets of the tiles in one block; the total into *total
__global__ void __launch_bounds__(1024) k_tile_offsets(int64_t ntiles, const int32_t* __restrict__ cnt,
                                                       int64_t* __restrict__ off, int64_t* __restrict__ total) {
    __shared__ int64_t sw[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t per = (ntiles + 1023) / 1024, a = per * threadIdx.x, b = a + per < ntiles ? a + per : ntiles;
    int64_t s = 0;
    for (int64_t i = a; i < b; ++i) s += cnt[i];
    int64_t x = s;
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sw[w] = x;
    __syncthreads();
    if (w == 0) {
        int64_t t = sw[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        sw[lane] = t;
    }
    __syncthreads();
    int64_t run = (w > 0 ? sw[w - 1] : 0) + x - s;
    for (int64_t i = a; i < b; ++i) {
        off[i] = run;
        run += cnt[i];
    }
    if (threadIdx.x == 1023) {
        off[ntiles] = run;
        *total = run;
    }
}

// the active tets of every tile that has any, in tet order
__global__ void __launch_bounds__(kTileThreads) k_compact(int64_t ngroups, int per_group, const uint8_t* __restrict__ bits,
                                                          const int64_t* __restrict__ off, int32_t* __restrict__ out) {
    const int64_t o0 = off[blockIdx.x];
    if (off[blockIdx.x + 1] == o0) return;
    __shared__ int wsum[kTileThreads / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t g0 = (int64_t)blockIdx.x * kTile + (int64_t)threadIdx.x * kTilePer;
    static_assert(kTilePer <= 8, "bits of one thread's groups in one word");
    unsigned long long b8 = 0;
    for (int j = 0; j < kTilePer; ++j)
        if (g0 + j < ngroups) b8 |= (unsigned long long)bits[g0 + j] << (8 * j);
    const int n = __popcll(b8);
    int x = n;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    int64_t pos = o0 + x - n;
    for (int k = 0; k < w; ++k) pos += wsum[k];
    while (b8) {
        const int bit = __ffsll((long long)b8) - 1;
        b8 &= b8 - 1;
        out[pos++] = (int32_t)((g0 + (bit >> 3)) * per_group + (bit & 7));
    }
}

// ---- numbering: vertices 0..nv-1, then (P2) edges, as one index range ----
__global__ void k_fill_keys(int64_t nv, int64_t ne, int32_t* __restrict__ kv, int32_t* __restrict__ ke) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nv + ne; i += (int64_t)gridDim.x * blockDim.x) {
        if (i < nv) kv[i] = INT_MAX;
        else ke[i - nv] = INT_MAX;
    }
}

__global__ void k_first_touch(MeshView M, int64_t n_active, const int32_t* __restrict__ active, int p2,
                              int32_t* __restrict__ kv, int32_t* __restrict__ ke) {
    const int nl = p2 ? 10 : 4;
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n_active; r += (int64_t)gridDim.x * blockDim.x) {
        int32_t v[4], e[6];
        mesh_tet(M, active[r], v, p2 ? e : nullptr);
        const int32_t base = (int32_t)(r * nl);
        for (int s = 0; s < 4; ++s) atomicMin(&kv[v[s]], base + s);
        if (p2)
            for (int s = 0; s < 6; ++s) atomicMin(&ke[e[s]], base + 4 + s);
    }
}

__global__ void k_mark_owned(int64_t nv, int64_t ne, const int32_t* __restrict__ kv, const int32_t* __restrict__ ke,
                             int32_t* __restrict__ owned) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nv + ne; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t k = i < nv ? kv[i] : ke[i - nv];
        if (k != INT_MAX) owned[k] = 1;
    }
}

__global__ void k_assign(int64_t nv, int64_t ne, const int32_t* __restrict__ kv, const int32_t* __restrict__ ke,
                         const int32_t* __restrict__ rank, int32_t* __restrict__ dv, int32_t* __restrict__ de) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nv + ne; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t k = i < nv ? kv[i] : ke[i - nv];
        const int32_t d = k != INT_MAX ? rank[k] : -1;
        if (i < nv) dv[i] = d;
        else de[i - nv] = d;
    }
}

__global__ void k_loc2glo(MeshView M, int64_t n_active, const int32_t* __restrict__ active, int p2,
                          const int32_t* __restrict__ dv, const int32_t* __restrict__ de, int32_t* __restrict__ l2g) {
    const int nl = p2 ? 10 : 4;
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n_active; r += (int64_t)gridDim.x * blockDim.x) {
        int32_t v[4], e[6];
        mesh_tet(M, active[r], v, p2 ? e : nullptr);
        for (int s = 0; s < 4; ++s) l2g[r * nl + s] = dv[v[s]];
        if (p2)
            for (int s = 0; s < 6; ++s) l2g[r * nl + 4 + s] = de[e[s]];
    }
}

int number_from_active(Context* c, int p2) {
    const MeshView& M = c->mesh;
    const int nl = p2 ? 10 : 4;
    const int64_t na = c->n_active, ne = p2 ? M.ne : 0;
    if (na * nl >= INT_MAX) return set_err(c, TF_ERR_CAPACITY, "too many active tets for 32-bit DOF keys");
    TimedLaunch tl(c, TF_K_NUMBER);
    TF_TRY(ensure(c, c->keys_v, (size_t)M.nv));
    TF_TRY(ensure(c, c->dof_vert, (size_t)M.nv));
    if (p2) {
        TF_TRY(ensure(c, c->keys_e, (size_t)M.ne));
        TF_TRY(ensure(c, c->dof_edge, (size_t)M.ne));
    }
    const int64_t nkeys = na * nl;
    TF_TRY(ensure(c, c->owner, (size_t)nkeys + 1));
    TF_TRY(ensure(c, c->loc2glo, (size_t)(nkeys > 0 ? nkeys : 1) + 1));  // scan output, then loc2glo
    TF_CUDA(c, cudaMemsetAsync(c->owner.p, 0, sizeof(int32_t) * (size_t)(nkeys + 1), c->stream));
    k_fill_keys<<<grid_for(c, M.nv + ne), kBlock, 0, c->stream>>>(M.nv, ne, c->keys_v.p, c->keys_e.p);
    if (na > 0) {
        k_first_touch<<<grid_for(c, na), kBlock, 0, c->stream>>>(M, na, c->active.p, p2, c->keys_v.p, c->keys_e.p);
        ++c->launches;
    }
    k_mark_owned<<<grid_for(c, M.nv + ne), kBlock, 0, c->stream>>>(M.nv, ne, c->keys_v.p, c->keys_e.p, c->owner.p);
    c->launches += 2;
    int64_t ndofs = 0;
    TF_TRY(exclusive_scan_i32_to_i32(c, c->owner.p, c->loc2glo.p, nkeys, &ndofs));
    k_assign<<<grid_for(c, M.nv + ne), kBlock, 0, c->stream>>>(M.nv, ne, c->keys_v.p, c->keys_e.p, c->loc2glo.p,
                                                               c->dof_vert.p, c->dof_edge.p);
    ++c->launches;
    if (na > 0) {
        k_loc2glo<<<grid_for(c, na), kBlock, 0, c->stream>>>(M, na, c->active.p, p2, c->dof_vert.p,
                                                              p2 ? c->dof_edge.p : nullptr, c->loc2glo.p);
        ++c->launches;
    }
    TF_CUDA(c, cudaGetLastError());
    c->n_dofs = ndofs;
    c->fe = p2 ? TF_P2IF : TF_P1IF;
    ++c->dof_version;
    return TF_OK;
}

int distribute_dofs(Context* c, int fe, double dist) {
    if (!c->has_mesh || !c->has_ls) return set_err(c, TF_ERR_BAD_INPUT, "distribute_dofs: mesh and level set required");
    if (fe != TF_P1IF && fe != TF_P2IF) return set_err(c, TF_ERR_BAD_INPUT, "distribute_dofs: fe must be TF_P1IF or TF_P2IF");
    const MeshView& M = c->mesh;
    c->fe = 0;
    c->legacy_numbering = false;
    const bool brick = !M.explicit_mesh;
    const int per_group = brick ? 6 : 1;
    const int64_t ngroups = M.nt / per_group, ntiles = (ngroups + kTile - 1) / kTile;
    if (ntiles > INT_MAX) return set_err(c, TF_ERR_CAPACITY, "distribute_dofs: too many tets");
    TF_TRY(ensure(c, c->flags, (size_t)(ngroups > 0 ? ngroups : 1)));
    TF_TRY(ensure(c, c->scan_tmp, (size_t)(ntiles + 1 + (ntiles + 1) / 2 + 1)));
    int64_t* off = c->scan_tmp.p;
    int32_t* cnt = reinterpret_cast<int32_t*>(off + ntiles + 1);
    TF_CUDA(c, cudaMemsetAsync(c->status.p, 0, kStatusWords * sizeof(int), c->stream));
    {
        TimedLaunch tl(c, TF_K_CLASSIFY);
        DistTest D;
        D.dmag_ok = dist >= 0.;
        D.dmag = 0;
        if (D.dmag_ok) {
            std::memcpy(&D.dmag, &dist, sizeof(double));
            D.dmag &= 0x7fffffffffffffffull;
        }
        D.mixed_active = 0. <= dist;
        static const CubeMasks masks = cube_masks();
        if (ntiles > 0) {
            if (brick)
                k_classify<true><<<(unsigned)ntiles, kTileThreads, 0, c->stream>>>(M, ngroups, c->ls_vert.p, c->ls_edge.p, D,
                                                                                   masks, c->flags.p, cnt, c->status.p);
            else
                k_classify<false><<<(unsigned)ntiles, kTileThreads, 0, c->stream>>>(M, ngroups, c->ls_vert.p, c->ls_edge.p,
                                                                                    D, masks, c->flags.p, cnt, c->status.p);
            ++c->launches;
        }
        k_tile_offsets<<<1, 1024, 0, c->stream>>>(ntiles, cnt, off, reinterpret_cast<int64_t*>(c->status.p + 4));
        ++c->launches;
        TF_CUDA(c, cudaGetLastError());
        int st = 0;
        TF_TRY(sync_status(c, &st));
        if (st != 0)
            return set_err(c, st, "distance: level set is exactly zero at a node of a cut tet (tet " +
                                      std::to_string(c->h_status[1]) + ")");
        std::memcpy(&c->n_active, c->h_status + 4, sizeof(int64_t));
        if (c->n_active > INT32_MAX) return set_err(c, TF_ERR_CAPACITY, "scan total exceeds int32 range");
        TF_TRY(ensure(c, c->active, (size_t)(c->n_active > 0 ? c->n_active : 1)));
        if (c->n_active > 0) {
            k_compact<<<(unsigned)ntiles, kTileThreads, 0, c->stream>>>(ngroups, per_group, c->flags.p, off, c->active.p);
            ++c->launches;
            TF_CUDA(c, cudaGetLastError());
        }
    }
    return number_from_active(c, fe == TF_P2IF);
}

}  // namespace tf

// Surface forms M, A, C_n and the load vector in pair arithmetic (ff.cuh).
//
// The FP64 kernels k_assemble<NL> keep the FP64 pipe 85% busy: per quadrature
// point ~190 FP64 operations for the P2 basis and ~220 lane FMAs for the M and
// A sums, and GB300 issues FP64 at 1/64 of the FP32 rate.  These kernels keep
// the per-tet work in FP64 (GetTrafoTr, the lattice patch with its cut points
// and facet areas: the same code as k_assemble), split the per-tet results
// into float pairs, and run everything per point -- quadrature node, weight
// and its square root, the level-set normal, the projected gradients, the
// load function -- and the element sums on the FP32 pipe in pair arithmetic.
// The sums are formed in the FP64 kernels' point order and point groups; the
// results differ from them by rounding (pair arithmetic carries ~48
// significant bits), inside the 1e-12 row-scaled parity bound.  Covered: M, A,
// C_n (P1 and P2) and a constant or TF_RHS_SPHERE_XYZ load vector; LaplaceM
// and N_P1P1 run k_assemble<4>.  (Pair arithmetic for the per-tet work as
// well was measured slower: the cut points and facet areas then take more
// issue slots on few lanes than their FP64 form takes on the FP64 pipe.)

struct TablesFF {
    ff q2_node[7][3], q2_w[7];
    ff q3_node[15][4], q3_sw[15];
};
__constant__ TablesFF cTF;
static bool g_tables_ff_ready[64] = {false};

static ff host_split(double x) {
    const float h = (float)x;
    return ff{h, (float)(x - (double)h)};
}

static int ensure_tables_ff(Context* c) {
    if (c->device >= 0 && c->device < 64 && g_tables_ff_ready[c->device]) return TF_OK;
    Tables T;
    build_tables(T);
    TablesFF F;
    for (int i = 0; i < 7; ++i) {
        for (int j = 0; j < 3; ++j) F.q2_node[i][j] = host_split(T.q2_node[i][j]);
        F.q2_w[i] = host_split(T.q2_w[i]);
    }
    for (int i = 0; i < 15; ++i) {
        for (int j = 0; j < 4; ++j) F.q3_node[i][j] = host_split(T.q3_node[i][j]);
        F.q3_sw[i] = host_split(T.q3_sw[i]);
    }
    TF_CUDA(c, cudaMemcpyToSymbol(cTF, &F, sizeof(TablesFF)));
    if (c->device >= 0 && c->device < 64) g_tables_ff_ready[c->device] = true;
    return TF_OK;
}

// Per warp.  Point rows are padded to an odd number of pairs per lane (11 and
// 21): a lane's row starts 22 or 42 words after its neighbour's, so the lanes'
// 64-bit stores of one column fall in distinct banks, and the contraction's
// reads of one row (one point, ten columns) do too.
struct AsmPairPts {
    ff phi[32][11];  // sqrt(w) phi_i; n . grad(phi_i) sqrt(w) for the volume rule
    ff sg[32][21];   // [2 i + c]: sqrt(w) grad(phi_i) in an orthonormal basis of the tangent plane
};
struct AsmPairSmem {
    AsmPairPts p;
    ff gl[4][3], G[4][3], X[4][3], absdet;
    ff fb[16][3][4], fw[16];
    ff fx[32];  // sqrt(w) f(x_p)
};

// the unit normal grad(phi_h) / |grad(phi_h)| at barycentric b
__device__ __noinline__ void ff_normal(const AsmPairSmem& S, const ff b[4], ff n[3]) {
    ff v[3];
    ffacc nn;
    for (int r = 0; r < 3; ++r) {
        ffacc q;
        for (int k = 0; k < 4; ++k) q.add_prod(b[k], S.G[k][r]);
        v[r] = q.value();
        nn.add_prod(v[r], v[r]);
    }
    const ff inv = ff_rsqrt(nn.value());
    for (int r = 0; r < 3; ++r) n[r] = ff_mul(v[r], inv);
}

// a . b through one accumulator (42 operations where chained pair sums take 64)
__device__ __forceinline__ ff ff_dot3a(const ff a[3], const ff b[3]) {
    ffacc q;
    for (int c = 0; c < 3; ++c) q.add_prod(a[c], b[c]);
    return q.value();
}

// An orthonormal basis (t0, t1) of the plane of unit normal n (Duff, Burgess, Christensen, Hery, Kensler, Liani, Villemin,
// "Building an orthonormal basis, revisited", 2017): one reciprocal, 1 / (1 + |n_z|), in pairs by a Newton step.
__device__ __forceinline__ void ff_tangents(const ff n[3], ff t0[3], ff t1[3]) {
    const float sg = copysignf(1.f, n[2].h);
    const ff d = ff_add_f(ff_scale(n[2], sg), 1.f);
    const float r0 = __frcp_rn(d.h);
    const ff q = ff_mul_f(d, r0);
    const ff a = ff_scale(ff_fast_two_sum(r0, __fmul_rn(r0, __fsub_rn(__fsub_rn(1.f, q.h), q.l))), -sg);
    const ff xa = ff_mul(n[0], a), b = ff_mul(xa, n[1]);
    t0[0] = ff_add_f(ff_scale(ff_mul(xa, n[0]), sg), 1.f);
    t0[1] = ff_scale(b, sg);
    t0[2] = ff_scale(n[0], -sg);
    t1[0] = b;
    t1[1] = ff_add_f(ff_mul(ff_mul(n[1], a), n[1]), sg);
    t1[2] = ff_neg(n[1]);
}

__device__ __forceinline__ ff ff_dot3(const ff a[3], const ff b[3]) {
    return ff_fma(a[2], b[2], ff_fma(a[1], b[1], ff_mul(a[0], b[0])));
}

// TF_RHS_SPHERE_XYZ: c * y0 y1 y2 at the closest point y of the sphere
__device__ __noinline__ ff ff_rhs(const RhsPar& R, const ff x[3]) {
    if (R.kind == TF_RHS_CONST) return ff_split(R.p[0]);
    if (R.kind != TF_RHS_SPHERE_XYZ) return ff_of(0.f);
    ff d[3];
    for (int r = 0; r < 3; ++r) d[r] = ff_sub(x[r], ff_split(R.p[r]));
    const ff n2 = ff_dot3(d, d);
    const ff inv = ff_rsqrt(n2);
    const ff dist = ff_sub(ff_mul(n2, inv), ff_split(R.p[3]));
    const ff s = ff_mul(dist, inv);
    ff y[3];
    for (int r = 0; r < 3; ++r) y[r] = ff_sub(x[r], ff_mul(s, d[r]));
    return ff_mul(ff_mul(ff_mul(ff_split(R.p[4]), y[0]), y[1]), y[2]);
}

// The pair forms' per-tet data, one thread per tet: the tet geometry
// (GetTrafoTr and the level set's vertex gradients), the patch on the
// order-2 lattice, with the arithmetic of warp_tet_geometry and warp_patch
// done serially.  The FP64 work of a tet is then one thread's
// instead of a warp's with 4 to 25 lanes active, so that every FP64 warp
// instruction works for 32 tets (GB300 runs FP64 at 1/64 of the FP32 rate).
struct TetPrep {
    ff gl[4][3], G[4][3], X[4][3];
    ff fb[16][3][4], fw[16];
    double absdet;
    ff absdet_ff;
    int nf;
};
constexpr int64_t kPrepChunk = 1 << 18;  // tets per prep pass (about 0.6 GB of records)

// Sign of a lattice value from its bits (a comparison holds the FP64 pipe 64 cycles): -1, 0, 1; 0 for NaN.
__device__ __forceinline__ int lat_sign(double x) {
    const long long b = __double_as_longlong(x);
    const unsigned long long m = (unsigned long long)b & 0x7fffffffffffffffull;
    return m == 0ull || m > 0x7ff0000000000000ull ? 0 : b < 0 ? -1 : 1;
}

// the lattice's negative and positive values as bits
__device__ __forceinline__ void lat_signs(const double lat[10], unsigned& neg, unsigned& pos) {
    neg = pos = 0u;
#pragma unroll
    for (int k = 0; k < 10; ++k) {
        const int s = lat_sign(lat[k]);
        neg |= (s < 0 ? 1u : 0u) << k;
        pos |= (s > 0 ? 1u : 0u) << k;
    }
}
// sign pattern of a sub-tet: sum (s_k + 1) 3^k
__device__ __forceinline__ int lat_pattern(int sub, unsigned neg, unsigned pos) {
    int pat = 0;
#pragma unroll
    for (int k = 3; k >= 0; --k) {
        const int v = cT.lat_t[sub][k];
        pat = 3 * pat + 1 + (int)(pos >> v & 1u) - (int)(neg >> v & 1u);
    }
    return pat;
}

// the same for a sub-tet that differs between lanes
__device__ __forceinline__ int lat_pattern_tab(const Tables* __restrict__ T, int sub, unsigned neg, unsigned pos) {
    int pat = 0;
#pragma unroll
    for (int k = 3; k >= 0; --k) {
        const int v = __ldg(&T->lat_t[sub][k]);
        pat = 3 * pat + 1 + (int)(pos >> v & 1u) - (int)(neg >> v & 1u);
    }
    return pat;
}
// cut_point of a lattice edge that differs between lanes
__device__ __forceinline__ void cut_point_tab(const Tables* __restrict__ T, const double lat[10], int k, double out[4]) {
    const int a = __ldg(&T->edge_a[k]), b = __ldg(&T->edge_b[k]);
    const double la = lat[a], t = __ddiv_rn(la, __dsub_rn(la, lat[b])), s = __dsub_rn(1.0, t);
    // lattice coordinates are 0, 1/2 and 1: the products are s, s/2, t, t/2 and 0, exactly, and at most two
    // coordinates have both (12 FP64 operations as a plain combination)
    const double hs = 0.5 * s, ht = 0.5 * t;
    for (int c = 0; c < 4; ++c) {
        const int ia = __double2hiint(__ldg(&T->lat_v[a][c])), ib = __double2hiint(__ldg(&T->lat_v[b][c]));
        const double u = ia == 0 ? 0. : ia == 0x3ff00000 ? s : hs, v = ib == 0 ? 0. : ib == 0x3ff00000 ? t : ht;
        out[c] = ia != 0 && ib != 0 ? __dadd_rn(u, v) : ia != 0 ? u : v;
    }
}

// The loops over lattice edges, sub-tets, facets and vertices stay rolled in
// the kernels below: unrolled, 150 to 190 KB of code ran from L2.
__global__ void __launch_bounds__(128) k_prep_tets(AsmArgs A) {
    TetPrep* const out = reinterpret_cast<TetPrep*>(A.prep);
    const int64_t n = A.prep_count ? *A.prep_count : A.c1 - A.c0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = A.c0 + (A.prep_order ? A.prep_order[i] : i);
        TetPrep& Q = out[r - A.c0];
        const int32_t t = A.active[r];
        int32_t v[4], e[6];
        TetGeom g;
        double ls10[10];
        mesh_tet_points(A.M, t, v, e, g.X);
        for (int k = 0; k < 4; ++k) ls10[k] = A.lsv[v[k]];
        for (int k = 0; k < 6; ++k) ls10[4 + k] = A.lse[e[k]];
        // warp_tet_geometry, lane by lane
        double Ms[9], Cs[9];
        for (int l = 0; l < 9; ++l) {
            const int rr = l / 3, c = l % 3;
            Ms[l] = g.X[c + 1][rr] - g.X[0][rr];
        }
        for (int l = 0; l < 9; ++l) {
            const int rr = l / 3, c = l % 3;
            const int r1 = (rr + 1) % 3, r2 = (rr + 2) % 3, c1 = (c + 1) % 3, c2 = (c + 2) % 3;
            Cs[l] = Ms[3 * r1 + c1] * Ms[3 * r2 + c2] - Ms[3 * r1 + c2] * Ms[3 * r2 + c1];
        }
        const double d = Ms[0] * Cs[0] + Ms[1] * Cs[1] + Ms[2] * Cs[2];
        const double inv = 1.0 / d;
        for (int vv = 0; vv < 4; ++vv)
            for (int rr = 0; rr < 3; ++rr)
                g.gl[vv][rr] = vv == 0 ? (-(Cs[3 * rr] * inv) - Cs[3 * rr + 1] * inv) - Cs[3 * rr + 2] * inv
                                       : Cs[3 * rr + vv - 1] * inv;
        g.absdet = fabs(d);
        for (int vv = 0; vv < 4; ++vv)
            for (int rr = 0; rr < 3; ++rr) {
                double sum = 0.;
                for (int i = 0; i < 4; ++i) sum += ls10[i] * ((i == vv ? 3. : -1.) * g.gl[i][rr]);
                for (int k = 0; k < 6; ++k) {
                    const int ea = ev0(k), eb = ev1(k);
                    if (eb == vv) sum += ls10[4 + k] * (4. * g.gl[ea][rr]);
                    if (ea == vv) sum += ls10[4 + k] * (4. * g.gl[eb][rr]);
                }
                g.G[vv][rr] = sum;
            }
        // warp_patch, lane by lane: cut points of the lattice edges, the sub-tets' facets in order
        double lat[10];
        for (int k = 0; k < 10; ++k) lat[cP2OnLat[k]] = ls10[k];
        unsigned neg, pos;
        lat_signs(lat, neg, pos);
        // every lane walks its own list of cut edges, then of facets (bit 2 s + f: facet f of sub-tet s), so lanes
        // with different patterns stay in step
        double cut[25][4];
        unsigned cuts = 0u;
#pragma unroll
        for (int k = 0; k < 25; ++k) {
            const int a = cT.edge_a[k], b = cT.edge_b[k];
            cuts |= (((neg >> a & pos >> b) | (pos >> a & neg >> b)) & 1u) << k;
        }
#pragma unroll 1
        for (unsigned m = cuts; m; m &= m - 1u) {
            const int k = __ffs((int)m) - 1;
            cut_point_tab(A.tab, lat, k, cut[k]);
        }
        unsigned facets = 0u;
#pragma unroll 1
        for (int sub = 0; sub < 8; ++sub) {
            const int nfs = __ldg(&A.tab->pat_nf[lat_pattern(sub, neg, pos)]);
            if (nfs < 0) set_status(A.status, TF_ERR_ZERO_PATTERN, t);
            facets |= (nfs > 1 ? 3u : nfs > 0 ? 1u : 0u) << (2 * sub);
        }
        int nf = 0;
#pragma unroll 1
        for (unsigned m = facets; m; m &= m - 1u, ++nf) {
            const int sub = (__ffs((int)m) - 1) >> 1, f = (__ffs((int)m) - 1) & 1;
            const int pat = lat_pattern_tab(A.tab, sub, neg, pos);
            double w[3][3];
#pragma unroll 1
            for (int j = 0; j < 3; ++j) {
                const int ext = __ldg(&A.tab->pat_f[pat][f][j]);
                double b[4];
                if (ext < 4) {
                    const int Lv = __ldg(&A.tab->lat_t[sub][ext]);
                    for (int c = 0; c < 4; ++c) b[c] = __ldg(&A.tab->lat_v[Lv][c]);
                } else {
                    const int id = __ldg(&A.tab->ledge[sub][ext - 4]);
                    for (int c = 0; c < 4; ++c) b[c] = cut[id][c];
                }
                for (int c = 0; c < 4; ++c) Q.fb[nf][j][c] = ff_split(b[c]);
                for (int rr = 0; rr < 3; ++rr)
                    w[j][rr] = g.X[0][rr] * b[0] + g.X[1][rr] * b[1] + g.X[2][rr] * b[2] + g.X[3][rr] * b[3];
            }
            double u[3], vq[3];
            for (int rr = 0; rr < 3; ++rr) {
                u[rr] = w[1][rr] - w[0][rr];
                vq[rr] = w[2][rr] - w[0][rr];
            }
            const double c0 = u[1] * vq[2] - u[2] * vq[1], c1 = u[2] * vq[0] - u[0] * vq[2],
                         c2 = u[0] * vq[1] - u[1] * vq[0];
            Q.fw[nf] = ff_split(sqrt(c0 * c0 + c1 * c1 + c2 * c2) * (__ldg(&A.tab->pat_bnd[pat]) ? 0.5 : 1.0));
        }
        Q.nf = nf;
        Q.absdet = g.absdet;
        Q.absdet_ff = ff_split(g.absdet);
#pragma unroll 1
        for (int vv = 0; vv < 4; ++vv)
            for (int c = 0; c < 3; ++c) {
                Q.gl[vv][c] = ff_split(g.gl[vv][c]);
                Q.G[vv][c] = ff_split(g.G[vv][c]);
                Q.X[vv][c] = ff_split(g.X[vv][c]);
            }
    }
}

__global__ void __launch_bounds__(32 * kAsmWarps) k_assemble_p2_pair(AsmArgs A) {
    constexpr int NL = 10, NSYM = 55, EPL = 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    AsmPairSmem& S = reinterpret_cast<AsmPairSmem*>(smem_raw)[wib];
    const bool wantM = A.forms & (1u << TF_FORM_M), wantA = A.forms & (1u << TF_FORM_A);
    const bool wantC = A.forms & (1u << TF_FORM_CN);
    const bool wantF = A.rhs.kind != TF_RHS_NONE;
    const int64_t nwarps = (int64_t)gridDim.x * kAsmWarps;

    const TetPrep* const prep = reinterpret_cast<const TetPrep*>(A.prep);
    for (int64_t r = A.c0 + (int64_t)blockIdx.x * kAsmWarps + wib; r < A.c1; r += nwarps) {
        // the tet's record (k_prep_tets): gl, G, X, |det| and the facets as pairs
        const TetPrep& Q = prep[r - A.c0];
        const int nf = Q.nf;
        for (int k = lane; k < 37; k += 32) {
            const int m = k / 12, v3 = (k % 12) / 3, c = k % 3;
            if (k == 36)
                S.absdet = Q.absdet_ff;
            else
                (m == 0 ? S.gl : m == 1 ? S.G : S.X)[v3][c] = (m == 0 ? Q.gl : m == 1 ? Q.G : Q.X)[v3][c];
        }
        for (int k = lane; k < 13 * nf; k += 32) {
            const int f = k / 13, j = k % 13;
            if (j == 12)
                S.fw[f] = Q.fw[f];
            else
                S.fb[f][j >> 2][j & 3] = Q.fb[f][j >> 2][j & 3];
        }
        __syncwarp();
        AsmPairPts& P = S.p;

        ffacc accM[EPL], accA[EPL], accF;
        const int npts = 7 * nf;
        for (int base = 0; base < npts; base += 32) {
            const int p = base + lane;
            if (p < npts) {
                const int f = p / 7, q = p - 7 * (p / 7);
                ff b[4];
                for (int c = 0; c < 4; ++c) {
                    ffacc v;
                    for (int j = 0; j < 3; ++j) v.add_prod(S.fb[f][j][c], cTF.q2_node[q][j]);
                    b[c] = v.value();
                }
                const ff sw = ff_sqrt(ff_mul(S.fw[f], cTF.q2_w[q]));
                ff n[3];
                ff_normal(S, b, n);
                // The basis loops are kept rolled (their operands in L1-resident local
                // memory): unrolled, the per-point pair code overflows the instruction cache.
                // The projected gradients lie in the tangent plane: two components in a basis of it
                // instead of three take a third off the A sums and the gradient rows (forms of the
                // P2 sphere 96^3 1,740 -> 1,622 us; A differs from the FP64 kernel by 1.6e-14 in the
                // norm, 2.4e-14 before).
                ff pg[4][2], q4[4];
                {
                    ff t0[3], t1[3];
                    ff_tangents(n, t0, t1);
#pragma unroll 1
                    for (int k = 0; k < 4; ++k) {
                        pg[k][0] = ff_mul(sw, ff_dot3a(S.gl[k], t0));
                        pg[k][1] = ff_mul(sw, ff_dot3a(S.gl[k], t1));
                        q4[k] = ff_scale(b[k], 4.f);
                    }
                }
#pragma unroll 1
                for (int i = 0; i < 10; ++i) {
                    // vertex i: phi = b_i (2 b_i - 1), grad = (4 b_i - 1) grad(b_i);
                    // edge (a, c): phi = 4 b_a b_c, grad = 4 b_c grad(b_a) + 4 b_a grad(b_c)
                    const int a = i < 4 ? i : ev0(i - 4), c2 = i < 4 ? i : ev1(i - 4);
                    const ff ph = i < 4 ? ff_mul(b[a], ff_add_f(ff_scale(b[a], 2.f), -1.f)) : ff_mul(q4[a], b[c2]);
                    P.phi[lane][i] = ff_mul(sw, ph);
                    const ff fa = i < 4 ? ff_add_f(q4[a], -1.f) : q4[c2];
                    for (int c = 0; c < 2; ++c) {
                        const ff t = ff_mul(fa, pg[a][c]);
                        P.sg[lane][2 * i + c] = i < 4 ? t : ff_fma(q4[a], pg[c2][c], t);
                    }
                }
                if (wantF) {
                    ff x[3];
                    for (int c = 0; c < 3; ++c) {
                        ffacc v;
                        for (int k = 0; k < 4; ++k) v.add_prod(b[k], S.X[k][c]);
                        x[c] = v.value();
                    }
                    S.fx[lane] = ff_mul(sw, ff_rhs(A.rhs, x));
                }
            }
            __syncwarp();
            const int cnt = min(32, npts - base);
            // entries k0 = lane and k1 = lane + 32 in one pass (lanes past the 55th entry repeat
            // the last one and do not store it)
            const int k1 = min(lane + 32, NSYM - 1);
            const int i0 = cT.sym_i[lane], j0 = cT.sym_j[lane], i1 = cT.sym_i[k1], j1 = cT.sym_j[k1];
            for (int pp = 0; pp < cnt; ++pp) {
                if (wantM) {
                    accM[0].add_prod(P.phi[pp][j0], P.phi[pp][i0]);
                    accM[1].add_prod(P.phi[pp][j1], P.phi[pp][i1]);
                }
                if (wantA)
                    for (int c = 0; c < 2; ++c) {
                        accA[0].add_prod(P.sg[pp][2 * j0 + c], P.sg[pp][2 * i0 + c]);
                        accA[1].add_prod(P.sg[pp][2 * j1 + c], P.sg[pp][2 * i1 + c]);
                    }
            }
            if (wantF && lane < 30) {  // 10 rows x 3 point groups (combined after the last chunk)
                const int i = lane % 10;
                for (int pp = lane / 10; pp < cnt; pp += 3) accF.add_prod(S.fx[pp], P.phi[pp][i]);
            }
            __syncwarp();
        }
        ff Fv = ff_of(0.f);
        if (wantF) {  // point groups (g0 + g1) + g2
            const ff f0 = accF.value();
            const ff f1{__shfl_down_sync(0xffffffffu, f0.h, 10), __shfl_down_sync(0xffffffffu, f0.l, 10)};
            const ff f2{__shfl_down_sync(0xffffffffu, f0.h, 20), __shfl_down_sync(0xffffffffu, f0.l, 20)};
            Fv = ff_add(ff_add(f0, f1), f2);
        }
        ffacc accC[EPL];
        if (wantC) {
            // normal-gradient volume stabilisation on the 15-point Quad5 rule
            if (lane < 15) {
                ff b[4];
                for (int c = 0; c < 4; ++c) b[c] = cTF.q3_node[lane][c];
                ff n[3];
                ff_normal(S, b, n);
                ff ng[4];
                for (int k = 0; k < 4; ++k) ng[k] = ff_mul(cTF.q3_sw[lane], ff_dot3(n, S.gl[k]));
                for (int i = 0; i < 4; ++i) P.phi[lane][i] = ff_mul(ff_add_f(ff_scale(b[i], 4.f), -1.f), ng[i]);
                for (int k = 0; k < 6; ++k) {
                    const int a = ev0(k), c2 = ev1(k);
                    P.phi[lane][4 + k] = ff_scale(ff_fma(b[c2], ng[a], ff_mul(b[a], ng[c2])), 4.f);
                }
            }
            __syncwarp();
            const int k1 = min(lane + 32, NSYM - 1);
            const int i0 = cT.sym_i[lane], j0 = cT.sym_j[lane], i1 = cT.sym_i[k1], j1 = cT.sym_j[k1];
            for (int pp = 0; pp < 15; ++pp) {
                accC[0].add_prod(P.phi[pp][j0], P.phi[pp][i0]);
                accC[1].add_prod(P.phi[pp][j1], P.phi[pp][i1]);
            }
            __syncwarp();
        }
        for (int qq = 0; qq < EPL; ++qq) {
            const int k = lane + 32 * qq;
            if (k >= NSYM) break;
            if (wantM) A.elem[((int64_t)TF_FORM_M * A.n_active + r) * NSYM + k] = ff_to_double(accM[qq].value());
            if (wantA) A.elem[((int64_t)TF_FORM_A * A.n_active + r) * NSYM + k] = ff_to_double(accA[qq].value());
            if (wantC)
                A.elem[((int64_t)TF_FORM_CN * A.n_active + r) * NSYM + k] =
                    ff_to_double(ff_mul(accC[qq].value(), S.absdet));
        }
        if (wantF && lane < NL) A.elem_rhs[r * NL + lane] = ff_to_double(Fv);
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// P1 forms M, A, C_n and the load vector in pair arithmetic (k_assemble_p1_pair).
// The tets whose level set is not linear: the normal, the projected gradients
// and the 15-point volume rule run per point; a warp takes a tet of the list
// that k_assemble_p1_linear left.
// Per point (node, weight and its square root, normal, gradients, load
// function) and every sum over points run in pair arithmetic; the point
// groups of the sums are those of k_assemble<4> (entries on 3 groups of
// 10 lanes, the load vector on 8 groups of 4).
// ---------------------------------------------------------------------------
struct AsmPair1Pts {
    ff phi[32][5];  // sqrt(w) b_i; n . grad(b_i) sqrt(w_q) for the volume rule (odd pitch: no bank conflicts)
    ff sg[32][13];  // [3 i + c]: sqrt(w) (I - n n^T) grad(b_i)
};
struct AsmPair1Smem {
    AsmPair1Pts p;
    ff gl[4][3], G[4][3], X[4][3];
    ff fb[16][3][4], fw[16];
    ff fx[32];  // sqrt(w) f(x_p)
};

__device__ __forceinline__ ff ff_shfl_down(ff a, int d) {
    return ff{__shfl_down_sync(0xffffffffu, a.h, d), __shfl_down_sync(0xffffffffu, a.l, d)};
}

__device__ __noinline__ void ff_normal1(const ff (*G)[3], const ff b[4], ff n[3]) {
    ff v[3];
    for (int r = 0; r < 3; ++r) {
        v[r] = ff_mul(b[0], G[0][r]);
        for (int k = 1; k < 4; ++k) v[r] = ff_fma(b[k], G[k][r], v[r]);
    }
    const ff nn = ff_fma(v[2], v[2], ff_fma(v[1], v[1], ff_mul(v[0], v[0])));
    const ff inv = ff_rsqrt(nn);
    for (int r = 0; r < 3; ++r) n[r] = ff_mul(v[r], inv);
}

__global__ void __launch_bounds__(32 * kAsmWarps) k_assemble_p1_pair(AsmArgs A) {
    constexpr int NL = 4, NSYM = 10;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    AsmPair1Smem& S = reinterpret_cast<AsmPair1Smem*>(smem_raw)[wib];
    const bool wantM = A.forms & (1u << TF_FORM_M), wantA = A.forms & (1u << TF_FORM_A);
    const bool wantC = A.forms & (1u << TF_FORM_CN);
    const bool wantF = A.rhs.kind != TF_RHS_NONE;
    const int64_t nwarps = (int64_t)gridDim.x * kAsmWarps;
    const TetPrep* const prep = reinterpret_cast<const TetPrep*>(A.prep);
    const int64_t n = *A.prep_count;
    for (int64_t i = (int64_t)blockIdx.x * kAsmWarps + wib; i < n; i += nwarps) {
        const int64_t r = A.c0 + A.prep_order[i];
        // the tet's record (k_prep_tets) into shared memory
        const TetPrep& Q = prep[r - A.c0];
        const int nf = Q.nf;
        const double absdet = Q.absdet;
        for (int k = lane; k < 36; k += 32) {
            const int m = k / 12, v3 = (k % 12) / 3, c = k % 3;
            (m == 0 ? S.gl : m == 1 ? S.G : S.X)[v3][c] = (m == 0 ? Q.gl : m == 1 ? Q.G : Q.X)[v3][c];
        }
        for (int k = lane; k < 13 * nf; k += 32) {
            const int f = k / 13, j = k % 13;
            if (j == 12)
                S.fw[f] = Q.fw[f];
            else
                S.fb[f][j >> 2][j & 3] = Q.fb[f][j >> 2][j & 3];
        }
        __syncwarp();
        AsmPair1Pts& P = S.p;

        ffacc accM, accA, accF;
        const int grp = lane / 10, k10 = lane % 10;
        int ei, ej;
        sym_entry(4, k10, ei, ej);
        const int npts = 7 * nf;
        for (int base = 0; base < npts; base += 32) {
            const int p = base + lane;
            if (p < npts) {
                const int f = p / 7, q = p - 7 * (p / 7);
                ff b[4];
                for (int c = 0; c < 4; ++c)
                    b[c] = ff_fma(S.fb[f][2][c], cTF.q2_node[q][2],
                                  ff_fma(S.fb[f][1][c], cTF.q2_node[q][1], ff_mul(S.fb[f][0][c], cTF.q2_node[q][0])));
                const ff w = ff_mul(S.fw[f], cTF.q2_w[q]);
                const ff sw = ff_sqrt(w);
                for (int i = 0; i < 4; ++i) P.phi[lane][i] = ff_mul(sw, b[i]);
                ff n[3];
                ff_normal1(S.G, b, n);
#pragma unroll 1
                for (int k = 0; k < 4; ++k) {
                    const ff ng = ff_dot3(n, S.gl[k]);
                    for (int c = 0; c < 3; ++c) P.sg[lane][3 * k + c] = ff_mul(sw, ff_sub(S.gl[k][c], ff_mul(ng, n[c])));
                }
                if (wantF) {
                    ff x[3];
                    for (int c = 0; c < 3; ++c)
                        x[c] = ff_fma(b[3], S.X[3][c],
                                      ff_fma(b[2], S.X[2][c], ff_fma(b[1], S.X[1][c], ff_mul(b[0], S.X[0][c]))));
                    S.fx[lane] = ff_mul(sw, ff_rhs(A.rhs, x));
                }
            }
            __syncwarp();
            const int cnt = min(32, npts - base);
            if (grp < 3) {
                for (int pp = grp; pp < cnt; pp += 3) {
                    if (wantM) accM.add_prod(P.phi[pp][ej], P.phi[pp][ei]);
                    if (wantA) {
                        accA.add_prod(P.sg[pp][3 * ej], P.sg[pp][3 * ei]);
                        accA.add_prod(P.sg[pp][3 * ej + 1], P.sg[pp][3 * ei + 1]);
                        accA.add_prod(P.sg[pp][3 * ej + 2], P.sg[pp][3 * ei + 2]);
                    }
                }
            }
            if (wantF)
                for (int pp = lane >> 2; pp < cnt; pp += 8) accF.add_prod(S.fx[pp], P.phi[pp][lane & 3]);
            __syncwarp();
        }
        // point groups: entries (g0 + g1) + g2, the load vector a tree over 8 groups
        ff vM = accM.value(), vA = accA.value(), vF = accF.value();
        vM = ff_add(ff_add(vM, ff_shfl_down(vM, 10)), ff_shfl_down(vM, 20));
        vA = ff_add(ff_add(vA, ff_shfl_down(vA, 10)), ff_shfl_down(vA, 20));
        vF = ff_add(vF, ff_shfl_down(vF, 16));
        vF = ff_add(vF, ff_shfl_down(vF, 8));
        vF = ff_add(vF, ff_shfl_down(vF, 4));
        double outC = 0.;
        if (wantC) {
            __syncwarp();
            if (lane < 15) {
                ff b[4];
                for (int c = 0; c < 4; ++c) b[c] = cTF.q3_node[lane][c];
                ff n[3];
                ff_normal1(S.G, b, n);
                for (int k = 0; k < 4; ++k) P.phi[lane][k] = ff_mul(cTF.q3_sw[lane], ff_dot3(n, S.gl[k]));
            }
            __syncwarp();
            ffacc accC;
            if (grp < 3)
                for (int pp = grp; pp < 15; pp += 3) accC.add_prod(P.phi[pp][ej], P.phi[pp][ei]);
            ff vC = accC.value();
            vC = ff_add(ff_add(vC, ff_shfl_down(vC, 10)), ff_shfl_down(vC, 20));
            outC = ff_to_double(vC) * absdet;
        }
        if (lane < NSYM) {
            if (wantM) A.elem[((int64_t)TF_FORM_M * A.n_active + r) * NSYM + lane] = ff_to_double(vM);
            if (wantA) A.elem[((int64_t)TF_FORM_A * A.n_active + r) * NSYM + lane] = ff_to_double(vA);
            if (wantC) A.elem[((int64_t)TF_FORM_CN * A.n_active + r) * NSYM + lane] = outC;
        }
        if (wantF && lane < NL) A.elem_rhs[r * NL + lane] = ff_to_double(vF);
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// P1 forms M, A, C_n and the load vector on tets whose level set is linear
// (every edge value the mean of its end values, bit for bit): G lanes per tet.
//
// The normal and the hat functions' surface gradients are constant, so
//   A_ij = |cut| sg_i . sg_j,  C_ij = |det| (sum_q w_q) dn_i dn_j,
// the hat functions are linear on the cut, so M is exact in closed form,
//   int phi_i phi_j = |facet| / 12 (S_i S_j + sum_k phi_i(v_k) phi_j(v_k)),
// S_i = sum_k phi_i(v_k), and a constant load's vector |facet| / 3 S_i: all on the
// cut of the whole tet, one or two triangles, where the quadrature took 7 points on
// each of up to 16 facets of the order-2 lattice.  Other loads keep that rule, the
// points of a facet summed into the moments sum_q w_q N_k(q) f(x_q) before they meet
// the basis.  Every lane walks the lists of its own tet's cut edges and facets, so
// lanes with different sign patterns stay in step.  Facets lie in one plane, so a facet's
// area is a constant of the tet times one 2 x 2 minor of barycentric differences.  Geometry, cut points and areas are FP64, everything per point
// and all sums pairs.
//
// Bound by the FP64 pipe (about 380 instructions per warp of 32 tets with a constant
// load, 500 with points, 64 cycles each; 47% busy) and, with points, the pair
// arithmetic.  Forms M, A, C_n of 126,800 cut tets (P1 sphere 128^3, prep and sort
// included): 868 -> 147 us with a constant load, 1,017 -> 354 with the closest-point
// load; 1,920 tets 143 -> 41 and 145 -> 71.  The warp per tet before formed 42 points on
// 64 lanes and its sums on 10 to 30 lanes, from 1.9 KB records of FP64 work unrolled to
// 152 KB of code.
//
// Tets whose level set is not linear go to `rest` (counted in *nrest, in the
// order of the threads up to the order of the warps' atomics).
// ---------------------------------------------------------------------------
// the closest-point load c y0 y1 y2 at centre + d: y = centre + R d / |d|
__device__ __forceinline__ ff ff_rhs_sphere(const ff ctr[3], ff R, ff amp, const ff d[3]) {
    ffacc n2;
    for (int r = 0; r < 3; ++r) n2.add_prod(d[r], d[r]);
    const ff s = ff_mul(R, ff_rsqrt(n2.value()));
    ff y[3];
    for (int r = 0; r < 3; ++r) y[r] = ff_fma(s, d[r], ctr[r]);
    return ff_mul(ff_mul(ff_mul(amp, y[0]), y[1]), y[2]);
}

template <int G>
__device__ __forceinline__ ff lane_group_sum(ff a) {
#pragma unroll
    for (int o = 1; o < G; o <<= 1)
        a = ff_add(a, ff{__shfl_xor_sync(0xffffffffu, a.h, o), __shfl_xor_sync(0xffffffffu, a.l, o)});
    return a;
}

// |u x w| of the facet's edges, where the level set's gradient is too small or large to give the plane's normal
__device__ __noinline__ double p1_area2(const double (&X)[4][3], const double (&du)[3], const double (&dv)[3]) {
    double u[3], w[3];
    for (int rr = 0; rr < 3; ++rr) {
        u[rr] = du[0] * (X[1][rr] - X[0][rr]) + du[1] * (X[2][rr] - X[0][rr]) + du[2] * (X[3][rr] - X[0][rr]);
        w[rr] = dv[0] * (X[1][rr] - X[0][rr]) + dv[1] * (X[2][rr] - X[0][rr]) + dv[2] * (X[3][rr] - X[0][rr]);
    }
    const double c0 = u[1] * w[2] - u[2] * w[1], c1 = u[2] * w[0] - u[0] * w[2], c2 = u[0] * w[1] - u[1] * w[0];
    return sqrt(c0 * c0 + c1 * c1 + c2 * c2);
}

// linear level set on the tet: every edge value the mean of its end values, bit for bit
__device__ __forceinline__ bool p1_linear_ls(const double (&ls10)[10]) {
    bool lin = true;
    for (int k = 0; k < 6; ++k) {
        const double mean = __dmul_rn(0.5, __dadd_rn(ls10[ev0(k)], ls10[ev1(k)]));
        lin = lin && __double_as_longlong(mean) == __double_as_longlong(ls10[4 + k]);
    }
    return lin;
}
__device__ __forceinline__ bool p1_linear_tet(const AsmArgs& A, int32_t t, double (&lat)[10]) {
    int32_t v[4], e[6];
    mesh_tet(A.M, t, v, e);
    double ls10[10];
    for (int k = 0; k < 10; ++k) ls10[k] = k < 4 ? A.lsv[v[k]] : A.lse[e[k - 4]];
    for (int k = 0; k < 10; ++k) lat[cP2OnLat[k]] = ls10[k];
    return p1_linear_ls(ls10);
}

// lattice edges that a linear level set cuts at most (every sign pattern whose edge midpoints take the sign of
// equal ends; a value that rounds to zero only takes cuts away)
constexpr int kLinCuts = 13;

template <int G, int B>
__global__ void __launch_bounds__(128, B) k_assemble_p1_linear(AsmArgs A, int32_t* __restrict__ rest, int* __restrict__ nrest) {
    constexpr int NSYM = 10;
    const bool wantM = A.forms & (1u << TF_FORM_M), wantA = A.forms & (1u << TF_FORM_A);
    const bool wantC = A.forms & (1u << TF_FORM_CN);
    const bool wantF = A.rhs.kind != TF_RHS_NONE, constF = A.rhs.kind == TF_RHS_CONST;
    const int lane = threadIdx.x & 31, sub = lane % G;
    const int64_t n = A.c1 - A.c0;
    double s3 = 0.;  // the 15-point rule's weight sum
    for (int q = 0; q < 15; ++q) s3 += cT.q3_w[q];
    // tets for the general kernels; whole warps call
    auto leave = [&](bool yes, int32_t rel) {
        const unsigned m = __ballot_sync(0xffffffffu, yes);
        if (!m) return;
        int at = 0;
        if (lane == 0) at = atomicAdd(nrest, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (yes) rest[at + __popc(m & ((1u << lane) - 1u))] = rel;
    };
    // Blocks of kTets tets.  With a point rule the block's tets are taken in the order of their facet counts: the
    // lanes of a warp walk their facets in step, and the longest list sets the warp's time.
    constexpr int kTets = 128 / G;
    __shared__ int32_t order[kTets];
    __shared__ int bin[17];
    for (int64_t i0 = (int64_t)blockIdx.x * kTets; i0 < n; i0 += (int64_t)gridDim.x * kTets) {
        const int m = (int)(n - i0 < kTets ? n - i0 : kTets);
        if (wantF && !constF) {
            __syncthreads();
            if (threadIdx.x < 17) bin[threadIdx.x] = 0;
            __syncthreads();
            int nf = 0, at = 0;
            bool linear = false;
            if ((int)threadIdx.x < m) {
                double lat[10];
                linear = p1_linear_tet(A, A.active[A.c0 + i0 + threadIdx.x], lat);
                unsigned neg, pos;
                lat_signs(lat, neg, pos);
#pragma unroll 1
                for (int s8 = 0; s8 < 8; ++s8) nf += max(0, (int)__ldg(&A.tab->pat_nf[lat_pattern(s8, neg, pos)]));
                at = atomicAdd(&bin[nf], 1);
            }
            __syncthreads();
            if ((int)threadIdx.x < m) {
                for (int k = 0; k < nf; ++k) at += bin[k];
                order[at] = linear ? (int32_t)threadIdx.x : ~(int32_t)threadIdx.x;
            }
            __syncthreads();
        }
        const int slot = threadIdx.x / G;
        const int at = slot >= m ? -1 : wantF && !constF ? order[slot] : slot;
        const bool valid = at >= 0;
        if (wantF && !constF) leave(slot < m && at < 0 && sub == 0, (int32_t)i0 + ~at);
        const int32_t rel = !valid ? 0 : (int32_t)i0 + at;
        const int64_t r = A.c0 + rel;
        const int32_t t = valid ? A.active[r] : 0;
        double X[4][3], lat[10];
        bool lin = valid;
        if (valid) {
            int32_t v[4], e[6];
            mesh_tet_points(A.M, t, v, e, X);
            double ls10[10];
            for (int k = 0; k < 10; ++k) ls10[k] = k < 4 ? A.lsv[v[k]] : A.lse[e[k - 4]];
            if (!(wantF && !constF)) lin = p1_linear_ls(ls10);
            for (int k = 0; k < 10; ++k) lat[cP2OnLat[k]] = ls10[k];
        }
        if (!(wantF && !constF)) leave(valid && !lin && sub == 0, rel);
        double gl[4][3], dn[4], absdet, per_minor = 0.;  // twice a facet's area per minor (c1, c2)
        int c1 = 1, c2 = 2;
        bool plane = false;
        if (lin) {
            double Ms[9], Cs[9];
            for (int l = 0; l < 9; ++l) Ms[l] = X[l % 3 + 1][l / 3] - X[0][l / 3];
            for (int l = 0; l < 9; ++l) {
                const int rr = l / 3, c = l % 3;
                const int r1 = (rr + 1) % 3, r2 = (rr + 2) % 3, c1 = (c + 1) % 3, c2 = (c + 2) % 3;
                Cs[l] = Ms[3 * r1 + c1] * Ms[3 * r2 + c2] - Ms[3 * r1 + c2] * Ms[3 * r2 + c1];
            }
            const double d = Ms[0] * Cs[0] + Ms[1] * Cs[1] + Ms[2] * Cs[2];
            const double inv = 1.0 / d;
            absdet = fabs(d);
            for (int vv = 1; vv < 4; ++vv)
                for (int rr = 0; rr < 3; ++rr) gl[vv][rr] = Cs[3 * rr + vv - 1] * inv;
            for (int rr = 0; rr < 3; ++rr) gl[0][rr] = (-gl[1][rr] - gl[2][rr]) - gl[3][rr];
            // the level set's gradient from the vertex values
            const double l0 = lat[cP2OnLat[0]];
            double g[3] = {0., 0., 0.}, dl[3];
            for (int vv = 1; vv < 4; ++vv) {
                dl[vv - 1] = lat[cP2OnLat[vv]] - l0;
                for (int rr = 0; rr < 3; ++rr) g[rr] += dl[vv - 1] * gl[vv][rr];
            }
            const double g2 = g[0] * g[0] + g[1] * g[1] + g[2] * g[2];
            const unsigned ge = (unsigned)(__double2hiint(g2) >> 20);
            plane = ge > 123u && ge < 1923u;  // 2^-900 < |g|^2 < 2^900: n is a unit vector
            const double inv_g = rsqrt_fp64(g2);
            for (int rr = 0; rr < 3; ++rr) g[rr] *= inv_g;
            for (int vv = 0; vv < 4; ++vv) dn[vv] = g[0] * gl[vv][0] + g[1] * gl[vv][1] + g[2] * gl[vv][2];
            // du x dv (of the coordinates 1..3) is parallel to the differences dl of the level set, and the area is
            // |d sum_c dn_c (du x dv)_c|: from the largest component alone, (du x dv)_k |d| |g| / |dl_k|, as
            // sum_c dn_c dl_c = |g|
            const double a0 = fabs(dl[0]), a1 = fabs(dl[1]), a2 = fabs(dl[2]);
            const long long i0 = __double_as_longlong(a0), i1 = __double_as_longlong(a1), i2 = __double_as_longlong(a2);
            const int k = i0 >= i1 && i0 >= i2 ? 0 : i1 >= i2 ? 1 : 2;
            c1 = k == 0 ? 1 : k == 1 ? 2 : 0;
            c2 = k == 0 ? 2 : k == 1 ? 0 : 1;
            per_minor = absdet * (g2 * inv_g) / (k == 0 ? a0 : k == 1 ? a1 : a2);
            // A needs the projected gradients' products
            if (wantA && sub == 0)
                for (int vv = 0; vv < 4; ++vv)
                    for (int c = 0; c < 3; ++c) gl[vv][c] -= dn[vv] * g[c];
        }
        // twice the area of a facet of barycentric corners b (components 1..3), as a pair
        auto area2 = [&](const double (&b)[3][3], float scale) {
            if (!plane) {
                double du[3], dv[3];
                for (int c = 0; c < 3; ++c) {
                    du[c] = b[1][c] - b[0][c];
                    dv[c] = b[2][c] - b[0][c];
                }
                return ff_scale(ff_split(p1_area2(X, du, dv)), scale);
            }
            // the minor of the two coordinates c1, c2
            auto pick = [](const double (&v)[3], int c) { return c == 0 ? v[0] : c == 1 ? v[1] : v[2]; };
            const double p0 = pick(b[0], c1), q0 = pick(b[0], c2);
            const double m = (pick(b[1], c1) - p0) * (pick(b[2], c2) - q0) - (pick(b[1], c2) - q0) * (pick(b[2], c1) - p0);
            return ff_scale(ff_split(fabs(m * per_minor)), scale);
        };
        unsigned neg = 0u, pos = 0u;
        ffacc accF[4];
        if (lin && sub == 0) {
            // M, A, C_n and a constant load: the cut of the whole tet, at most two triangles
            lat_signs(lat, neg, pos);
            int pat = 0;
            for (int k = 3; k >= 0; --k) pat = 3 * pat + 1 + (int)(pos >> cP2OnLat[k] & 1u) - (int)(neg >> cP2OnLat[k] & 1u);
            const int nf = __ldg(&A.tab->pat_nf[pat]);
            const float scale = __ldg(&A.tab->pat_bnd[pat]) ? 0.5f : 1.0f;
            if (nf < 0) set_status(A.status, TF_ERR_ZERO_PATTERN, t);
            ffacc accM[NSYM], accA;
#pragma unroll 1
            for (int f = 0; f < nf; ++f) {
                double b[3][3];
                ff p[4][4];
#pragma unroll 1
                for (int j = 0; j < 3; ++j) {
                    const int ext = __ldg(&A.tab->pat_f[pat][f][j]);
                    int va = ext, vb = ext;
                    double st = 1.0, tt = 0.0;
                    if (ext >= 4) {
                        va = ev0(ext - 4);
                        vb = ev1(ext - 4);
                        const double la = lat[cP2OnLat[va]], lb = lat[cP2OnLat[vb]];
                        tt = __ddiv_rn(la, __dsub_rn(la, lb));
                        st = __dsub_rn(1.0, tt);
                    }
                    const ff sf = ff_split(st), tf = ff_split(tt);
                    for (int c = 0; c < 4; ++c) {
                        p[j][c] = c == va ? sf : c == vb ? tf : ff_of(0.f);
                        if (c > 0) b[j][c - 1] = c == va ? st : c == vb ? tt : 0.0;
                    }
                }
                const ff fw = area2(b, scale);
                accA.add(fw);
                for (int c = 0; c < 4; ++c) p[3][c] = ff_add(ff_add(p[0][c], p[1][c]), p[2][c]);
                if (constF)
                    for (int c = 0; c < 4; ++c) accF[c].add_prod(fw, p[3][c]);
#pragma unroll 1
                for (int j = 0; j < 4; ++j) {
                    ff q[4];
                    for (int c = 0; c < 4; ++c) q[c] = p[j][c];
                    int k = 0;  // entry (a, c), a <= c, row by row
#pragma unroll
                    for (int a = 0; a < 4; ++a) {
                        const ff tq = ff_mul(fw, q[a]);
#pragma unroll
                        for (int c = a; c < 4; ++c) accM[k++].add_prod(tq, q[c]);
                    }
                }
            }
            const int64_t e = r * (NSYM / 2), form = A.n_active * (NSYM / 2);
            double2* const el = reinterpret_cast<double2*>(A.elem);
            if (wantM) {
#pragma unroll
                for (int k = 0; k < NSYM; k += 2)
                    el[TF_FORM_M * form + e + k / 2] = make_double2(ff_widen(accM[k].value()) * (1.0 / 24.0),
                                                                    ff_widen(accM[k + 1].value()) * (1.0 / 24.0));
            }
            if (wantA) {
                const double area = 0.5 * ff_widen(accA.value());
                double w[NSYM];
                int k = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = i; j < 4; ++j)
                        w[k++] = area * (gl[j][0] * gl[i][0] + gl[j][1] * gl[i][1] + gl[j][2] * gl[i][2]);
#pragma unroll
                for (int k = 0; k < NSYM; k += 2) el[TF_FORM_A * form + e + k / 2] = make_double2(w[k], w[k + 1]);
            }
            if (wantC) {
                const double s3d = s3 * absdet;
                double w[NSYM];
                int k = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = i; j < 4; ++j) w[k++] = s3d * (dn[j] * dn[i]);
#pragma unroll
                for (int k = 0; k < NSYM; k += 2) el[TF_FORM_CN * form + e + k / 2] = make_double2(w[k], w[k + 1]);
            }
        }
        if (lin && wantF && !constF) {
            // other loads: the 7-point rule on the facets of the order-2 lattice
            const ff ctr[3] = {ff_split(A.rhs.p[0]), ff_split(A.rhs.p[1]), ff_split(A.rhs.p[2])};
            const ff R = ff_split(A.rhs.p[3]), amp = ff_split(A.rhs.p[4]);
            ff Xf[4][3];
#pragma unroll 1
            for (int vv = 0; vv < 4; ++vv)
                for (int c = 0; c < 3; ++c) Xf[vv][c] = ff_sub(ff_split(X[vv][c]), ctr[c]);
            if (G > 1) lat_signs(lat, neg, pos);
            // the lattice edges cut and their points in this order; every lane walks its own list, so lanes with
            // different patterns stay in step
            unsigned cuts = 0u;
#pragma unroll
            for (int k = 0; k < 25; ++k) {
                const int a = cT.edge_a[k], b = cT.edge_b[k];
                cuts |= (((neg >> a & pos >> b) | (pos >> a & neg >> b)) & 1u) << k;
            }
            double cut[kLinCuts][4];
            int ncut = 0;
#pragma unroll 1
            for (unsigned m = cuts; m && ncut < kLinCuts; m &= m - 1u, ++ncut) {
                cut_point_tab(A.tab, lat, __ffs((int)m) - 1, cut[ncut]);
            }
            // the facets: bit 2 s + f is facet f of sub-tet s
            unsigned facets = 0u;
#pragma unroll 1
            for (int s8 = 0; s8 < 8; ++s8) {
                const int nfs = __ldg(&A.tab->pat_nf[lat_pattern(s8, neg, pos)]);
                if (nfs < 0) set_status(A.status, TF_ERR_ZERO_PATTERN, t);
                facets |= (nfs > 1 ? 3u : nfs > 0 ? 1u : 0u) << (2 * s8);
            }
            // a lane takes every G-th of them
            auto drop = [](unsigned m, int k) {
                for (; k > 0; --k) m &= m - 1u;
                return m;
            };
#pragma unroll 1
            for (unsigned m = drop(facets, sub); m; m = drop(m, G)) {
                const int s8 = (__ffs((int)m) - 1) >> 1, f = (__ffs((int)m) - 1) & 1;
                const int pat = lat_pattern_tab(A.tab, s8, neg, pos);
                const float scale = __ldg(&A.tab->pat_bnd[pat]) ? 0.5f : 1.0f;
                // corners: barycentric, as pairs p[j], and world coordinates from the centre Y[j]
                double b[3][3];
                ff p[3][4], Y[3][3];
#pragma unroll 1
                for (int j = 0; j < 3; ++j) {
                    const int ext = __ldg(&A.tab->pat_f[pat][f][j]);
                    double v[4];
                    if (ext < 4) {
                        const int lv = __ldg(&A.tab->lat_t[s8][ext]);
                        for (int c = 0; c < 4; ++c) v[c] = __ldg(&A.tab->lat_v[lv][c]);
                    } else {
                        const int id = __ldg(&A.tab->ledge[s8][ext - 4]);
                        const int at = min(__popc(cuts & ((1u << id) - 1u)), kLinCuts - 1);
                        for (int c = 0; c < 4; ++c) v[c] = cut[at][c];
                    }
                    ff pj[4];
                    for (int c = 0; c < 4; ++c) {
                        pj[c] = ff_split(v[c]);
                        p[j][c] = pj[c];
                        if (c > 0) b[j][c - 1] = v[c];
                    }
                    for (int c = 0; c < 3; ++c) {
                        ffacc y;
                        for (int k = 0; k < 4; ++k) y.add_prod(pj[k], Xf[k][c]);
                        Y[j][c] = y.value();
                    }
                }
                const ff fw = area2(b, scale);
                ffacc mom[3];
#pragma unroll 1
                for (int q = 0; q < 7; ++q) {
                    ff d[3];
                    for (int c = 0; c < 3; ++c) {
                        ffacc x;
                        for (int j = 0; j < 3; ++j) x.add_prod(Y[j][c], cTF.q2_node[q][j]);
                        d[c] = x.value();
                    }
                    const ff wf = ff_mul(cTF.q2_w[q], ff_rhs_sphere(ctr, R, amp, d));
                    for (int j = 0; j < 3; ++j) mom[j].add_prod(wf, cTF.q2_node[q][j]);
                }
                for (int j = 0; j < 3; ++j) {
                    const ff w = ff_mul(fw, mom[j].value());
                    for (int c = 0; c < 4; ++c) accF[c].add_prod(w, p[j][c]);
                }
            }
        }
        ff vF[4];
        for (int k = 0; k < 4; ++k) vF[k] = lane_group_sum<G>(accF[k].value());
        if (!lin || sub != 0) continue;
        if (wantF) {
            const double c = constF ? A.rhs.p[0] * (1.0 / 6.0) : 1.0;
            double2* const o = reinterpret_cast<double2*>(A.elem_rhs + r * 4);
            o[0] = make_double2(c * ff_widen(vF[0]), c * ff_widen(vF[1]));
            o[1] = make_double2(c * ff_widen(vF[2]), c * ff_widen(vF[3]));
        }
    }
}

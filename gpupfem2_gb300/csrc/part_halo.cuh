// part_halo.cuh - partitioned CG with halo rows (included by solvers.cu).
//
// k_pcg_part's sweeps wait, colour by colour, for other parts' boundary values, and a third
// grid-wide step per iteration publishes the boundary rows' direction.  Here each part also
// computes the few rows around it that its own rows depend on (the same arithmetic on the same
// inputs, so the same bits as their owner), and an iteration has no wait inside a sweep:
//   F rows: other parts' rows that the part's forward sweep reads, closed under the sweep's
//           dependencies (lower groups).  Their r lives here too: r -= alpha q with the owner's
//           q, which owners publish before the p.q reduction and which is read behind its
//           barrier.
//   Z rows: the neighbour rows of the part's rows (ring 1, whose p the SpMV reads), closed under
//           the backward sweep's dependencies (higher groups).  Their forward result t is either
//           computed here (F rows) or read once from the owner, polled on the pending marker.
// p on ring 1 follows from its z, so the direction needs no exchange.  Per iteration: SpMV;
// reduction of p.q; forward sweep; (IC(0): arrival at the t.t reduction;) t of the Z rows that
// are not F rows; backward sweep; reduction (IC(0): the wait alone).
//
// Local numbering of part k: its rows 0 .. np - 1 (Q order), then its halo rows by group, each
// group's rows as F only, F and Z, Z only.  Columns are local (16 bits), so no lookup or branch
// tells own entries from others'.
//
// What bounds it: FP64 issue of the rows (SpMV, sweeps) plus two reductions' latency.  Measured,
// us per iteration, k_pcg_part -> this kernel (same bits), cylinder pressure matrix:
//   125,364 rows: IC(0) 29.7 -> 21.8, ILU(0) 34.4 -> 22.5, mixed IC(0) 28.3 -> 19.0, Jacobi 16.1 -> 14.9
//   499,288 rows: IC(0) 43.1 -> 39.5, ILU(0) 45.2 -> 40.4, mixed IC(0) 34.1 -> 27.2, Jacobi 28.3 -> 24.9
#pragma once

namespace pf2 {

struct PartHalo {
    int P, ng;
    int R;                      // largest number of own rows
    int RL;                     // largest number of local rows (own + halo)
    const int* qs;              // own group starts (PartCg::qs)
    const int* hs;              // [(part * ng + group) * 4]: halo rows' F start, Z start, F end, Z end
    const int* hoff;            // P + 1: the parts' halo rows in hq
    const int* hq;              // halo row -> row in Q order
    const int* foff;            // P + 1: the parts' F rows in fl, fg (local index, row in Q order)
    const unsigned short* fl;
    const int* fg;
    const int* zoff;            // P + 1: the parts' Z rows that are not F rows in zl, zg
    const unsigned short* zl;
    const int* zg;
    const int* r1off;           // P + 1: the parts' ring-1 rows in r1
    const unsigned short* r1;   // local indices of ring-1 rows
    const int* ebase;           // P + 1: the parts' first entry
    const int* rp;              // part k: np + nh + 1 entry offsets at qs[k ng] + hoff[k] + k
    const unsigned char* dg;    // offset of the diagonal in the row's entries, at qs[k ng] + hoff[k]
    const unsigned char* pub;   // own rows: bit 0 q (and r) is read by another part, bit 1 t is
    const unsigned short* lcol; // local columns
    const int* qa;              // Q row -> row of A
    const double* val;
    const double* f;
    double* x;
    double* gq;                 // published q (r at the start and at refinements), Q order
    double* gt;                 // 2 n: published t, the sweeps alternate halves (pending markers)
    const float* val32;
    const float* f32;
    float* gq32;
    float* gt32;
};

template <class V> struct HaloVecs;
template <> struct HaloVecs<double> {
    __device__ static const double* val(const PartHalo& C) { return C.val; }
    __device__ static const double* f(const PartHalo& C) { return C.f; }
    __device__ static double* gq(const PartHalo& C) { return C.gq; }
    __device__ static double* gt(const PartHalo& C) { return C.gt; }
};
template <> struct HaloVecs<float> {
    __device__ static const float* val(const PartHalo& C) { return C.val32; }
    __device__ static const float* f(const PartHalo& C) { return C.f32; }
    __device__ static float* gq(const PartHalo& C) { return C.gq32; }
    __device__ static float* gt(const PartHalo& C) { return C.gt32; }
};

// A part in shared memory: r, p, q, t (z shares t's array; Jacobi / none: t = 1 / a_ii and z
// apart) over the local rows, the mixed solver's update d over the own rows, the reduction
// scratch, the rows' entry offsets and diagonals, the own rows' publication flags.  val, f and
// lcol point at the part's first entry.
template <class V>
struct HaloSm {
    V *r, *p, *q, *t, *z, *d;
    double* red;
    const int* rp;
    const unsigned char *dg, *pub;
    const V *val, *f;
    const unsigned short* lcol;
    const int* hq;   // the part's halo rows
    const int* hs;   // the part's group table
    const int* qs;   // the part's group starts
    int p0, np, nh, n, par;
    // the exchanged rows of this thread's first pass (fetches without a look-up load before them)
    int nf, f_l, f_g, nz, z_l, z_g;
};

__host__ __device__ constexpr size_t halo_vec_bytes(int R, int RL, bool tri, size_t vsz, bool mixed) {
    return ((size_t)(4 + (tri ? 0 : 1)) * RL * vsz + (mixed ? (size_t)R * vsz : 0) + 15) / 16 * 16;
}
__host__ __device__ constexpr size_t halo_smem_bytes(int R, int RL, bool tri, size_t vsz, bool mixed) {
    return (halo_vec_bytes(R, RL, tri, vsz, mixed) + sizeof(double) * 2 * kPartThreads +
            sizeof(int) * ((size_t)RL + 1) + (size_t)RL + (size_t)R + 15) / 16 * 16;
}

template <class V>
__device__ __forceinline__ HaloSm<V> halo_sm(const PartHalo& C, int n, unsigned char* base, bool tri, bool mixed) {
    HaloSm<V> S;
    const int k = blockIdx.x;
    S.n = n;
    S.qs = C.qs + k * C.ng;
    S.p0 = S.qs[0];
    S.np = S.qs[C.ng] - S.p0;
    const int h0 = C.hoff[k];
    S.nh = C.hoff[k + 1] - h0;
    S.hq = C.hq + h0;
    S.hs = C.hs + 4 * k * C.ng;
    S.par = 0;
    V* v = reinterpret_cast<V*>(base);
    S.r = v;
    S.p = v + C.RL;
    S.q = v + 2 * C.RL;
    S.t = v + 3 * C.RL;
    S.z = tri ? S.t : v + 4 * C.RL;
    S.d = mixed ? v + (tri ? 4 : 5) * C.RL : nullptr;
    S.red = reinterpret_cast<double*>(base + halo_vec_bytes(C.R, C.RL, tri, sizeof(V), mixed));
    int* rp = reinterpret_cast<int*>(S.red + 2 * kPartThreads);
    unsigned char* dg = reinterpret_cast<unsigned char*>(rp + C.RL + 1);
    unsigned char* pub = dg + C.RL;
    const int e0 = C.ebase[k];
    S.val = HaloVecs<V>::val(C) + e0;
    S.f = HaloVecs<V>::f(C) ? HaloVecs<V>::f(C) + e0 : nullptr;
    S.lcol = C.lcol + e0;
    const int nl = S.np + S.nh;
    const int* grp = C.rp + S.p0 + h0 + k;
    const unsigned char* gdg = C.dg + S.p0 + h0;
    for (int l = threadIdx.x; l <= nl; l += kPartThreads) rp[l] = __ldg(&grp[l]);
    for (int l = threadIdx.x; l < nl; l += kPartThreads) dg[l] = __ldg(&gdg[l]);
    for (int l = threadIdx.x; l < S.np; l += kPartThreads) pub[l] = __ldg(&C.pub[S.p0 + l]);
    S.rp = rp;
    S.dg = dg;
    S.pub = pub;
    const int f0 = C.foff[k], z0 = C.zoff[k];
    S.nf = C.foff[k + 1] - f0;
    S.nz = C.zoff[k + 1] - z0;
    S.f_l = S.f_g = S.z_l = S.z_g = 0;
    if ((int)threadIdx.x < S.nf) {
        S.f_l = C.fl[f0 + threadIdx.x];
        S.f_g = C.fg[f0 + threadIdx.x];
    }
    if ((int)threadIdx.x < S.nz) {
        S.z_l = C.zl[z0 + threadIdx.x];
        S.z_g = C.zg[z0 + threadIdx.x];
    }
    return S;
}

// Row in Q order of local row l.
template <class V>
__device__ __forceinline__ int halo_global(const HaloSm<V>& S, int l) {
    return l < S.np ? S.p0 + l : __ldg(&S.hq[l - S.np]);
}

// q = A p over the part's rows (part_spmv's arithmetic); the rows that are F rows elsewhere
// are published.  Returns the thread's p.q terms in FP64.
template <class V>
__device__ __forceinline__ double halo_spmv(const PartHalo& C, const HaloSm<V>& S) {
    V* gq = HaloVecs<V>::gq(C);
    double pq = 0.0;
    for (int l = threadIdx.x; l < S.np; l += kPartThreads) {
        const int s = S.rp[l], e = S.rp[l + 1];
        V acc = V(0);
        for (int k = s; k < e; ++k) acc += __ldg(&S.val[k]) * S.p[__ldg(&S.lcol[k])];
        S.q[l] = acc;
        if (S.pub[l] & 1) __stcg(&gq[S.p0 + l], acc);
        pq += (double)S.p[l] * (double)acc;
    }
    return pq;
}

// dst of the part's F rows from the published values (behind a grid barrier).
template <class V>
__device__ __forceinline__ void halo_fetch(const PartHalo& C, const HaloSm<V>& S, V* dst) {
    const V* gq = HaloVecs<V>::gq(C);
    if ((int)threadIdx.x < S.nf) dst[S.f_l] = __ldcg(&gq[S.f_g]);
    for (int i = threadIdx.x + kPartThreads, f0 = __ldg(&C.foff[blockIdx.x]); i < S.nf; i += kPartThreads)
        dst[__ldg(&C.fl[f0 + i])] = __ldcg(&gq[__ldg(&C.fg[f0 + i])]);
}

// r of the own rows published for the parts that hold them as F rows.
template <class V>
__device__ __forceinline__ void halo_publish_r(const PartHalo& C, const HaloSm<V>& S) {
    V* gq = HaloVecs<V>::gq(C);
    for (int l = threadIdx.x; l < S.np; l += kPartThreads)
        if (S.pub[l] & 1) __stcg(&gq[S.p0 + l], S.r[l]);
}

// s - sum_k f_k v[col_k] over the entries [k0, k1) (sweep_rest's chain of fused multiply-adds).
template <class V>
__device__ __forceinline__ V halo_rest(const HaloSm<V>& S, int k0, int k1, const V* v, V s) {
    for (int k = k0; k < k1; ++k) s = fma_rn(-__ldg(&S.f[k]), v[__ldg(&S.lcol[k])], s);
    return s;
}

// Forward sweep (part_fwd's arithmetic) over the own rows and the F rows, group by group, with
// r -= alpha q unless first.  Own t that is read elsewhere goes to this sweep's half of gt, and
// the other half, which every part has read before the last grid barrier, back to the marker.
// Returns the own rows' r.r (want_rr) and t.t terms.
template <bool IC, class V>
__device__ double2 halo_fwd(const PartHalo& C, HaloSm<V>& S, bool first, V alpha, bool want_rr) {
    V* gt = HaloVecs<V>::gt(C) + (size_t)S.par * S.n + S.p0;
    V* gt_next = HaloVecs<V>::gt(C) + (size_t)(S.par ^ 1) * S.n + S.p0;
    double rr = 0.0, tt = 0.0;
    for (int g = 0; g < C.ng; ++g) {
        const int g0 = S.qs[g] - S.p0, no = S.qs[g + 1] - S.p0 - g0;
        const int f0 = S.np + __ldg(&S.hs[4 * g]), nf = S.np + __ldg(&S.hs[4 * g + 2]) - f0;
        if ((int)threadIdx.x < no + nf) {
            const int l = (int)threadIdx.x < no ? g0 + threadIdx.x : f0 + threadIdx.x - no;
            const int k0 = S.rp[l], d = k0 + S.dg[l];
            prefetch_l1(&S.lcol[k0]);
            prefetch_l1(&S.f[k0]);
            prefetch_l1(&S.f[d]);
        }
        __syncthreads();  // the part's earlier groups are done
        for (int i = threadIdx.x; i < no + nf; i += kPartThreads) {
            const bool own = i < no;
            const int l = own ? g0 + i : f0 + i - no;
            const int k0 = S.rp[l], d = k0 + S.dg[l];
            V ra = S.r[l];
            if (!first) {
                ra -= alpha * S.q[l];
                S.r[l] = ra;
            }
            const V rest = halo_rest(S, k0, d, S.t, ra);
            const V v = IC ? rest * __ldg(&S.f[d]) : rest;
            S.t[l] = v;
            if (own) {
                if (S.pub[l] & 2) {
                    __stcg(&gt[l], v);
                    __stcg(&gt_next[l], Pending<V>::marker());
                }
                if (want_rr) rr += (double)ra * (double)ra;
                if (IC) tt += (double)v * (double)v;
            }
        }
    }
    return make_double2(rr, tt);
}

// t of the Z rows that are not F rows, from their owners (bounded polls; a wait that runs out
// records DEV_TIMEOUT and yields 0: the kernel returns at its next grid barrier).  The next
// forward sweep uses the other half of gt.
template <class V>
__device__ __forceinline__ void halo_fetch_t(const PartHalo& C, HaloSm<V>& S, int* err, int* rec) {
    const V* gt = HaloVecs<V>::gt(C) + (size_t)S.par * S.n;
    auto fetch = [&](int l, int j) {
        V v = *(volatile const V*)&gt[j];
        if (Pending<V>::bits(v) == Pending<V>::kBits && !wait_value(gt, j, v, err, rec, j)) v = V(0);
        S.t[l] = v;
    };
    if ((int)threadIdx.x < S.nz) fetch(S.z_l, S.z_g);
    for (int i = threadIdx.x + kPartThreads, z0 = __ldg(&C.zoff[blockIdx.x]); i < S.nz; i += kPartThreads)
        fetch(__ldg(&C.zl[z0 + i]), __ldg(&C.zg[z0 + i]));
    S.par ^= 1;
}

// Backward sweep (part_bwd's arithmetic) over the own rows and the Z rows: z = U^{-1} t in t's
// array.  Returns the own rows' r.z terms (want_rz).
template <class V>
__device__ double halo_bwd(const PartHalo& C, const HaloSm<V>& S, bool want_rz) {
    double rz = 0.0;
    for (int g = C.ng - 1; g >= 0; --g) {
        const int g0 = S.qs[g] - S.p0, no = S.qs[g + 1] - S.p0 - g0;
        const int z0 = S.np + __ldg(&S.hs[4 * g + 1]), nz = S.np + __ldg(&S.hs[4 * g + 3]) - z0;
        if ((int)threadIdx.x < no + nz) {
            const int l = (int)threadIdx.x < no ? g0 + threadIdx.x : z0 + threadIdx.x - no;
            const int d = S.rp[l] + S.dg[l];
            prefetch_l1(&S.lcol[d]);
            prefetch_l1(&S.f[d]);
            prefetch_l1(&S.f[S.rp[l + 1] - 1]);
        }
        __syncthreads();  // the part's later groups are done
        for (int i = threadIdx.x; i < no + nz; i += kPartThreads) {
            const bool own = i < no;
            const int l = own ? g0 + i : z0 + i - no;
            const int d = S.rp[l] + S.dg[l];
            const V v = halo_rest(S, d + 1, S.rp[l + 1], S.z, S.t[l]) * __ldg(&S.f[d]);
            S.z[l] = v;
            if (want_rz && own) rz += (double)S.r[l] * (double)v;
        }
    }
    return rz;
}

// p = z + beta p (first: p = z) on the own rows and ring 1.  No barrier inside; the SpMV that
// follows needs one.
template <class V>
__device__ __forceinline__ void halo_p_update(const PartHalo& C, const HaloSm<V>& S, V beta, bool first) {
    const int k = blockIdx.x;
    const int a0 = __ldg(&C.r1off[k]), nr = __ldg(&C.r1off[k + 1]) - a0;
    for (int i = threadIdx.x; i < S.np + nr; i += kPartThreads) {
        const int l = i < S.np ? i : (int)__ldg(&C.r1[a0 + i - S.np]);
        S.p[l] = first ? S.z[l] : fma_rn(beta, S.p[l], S.z[l]);
    }
}

// b - A x in FP64 for the part's row l (x from the global iterate in Q order).
template <class V>
__device__ __forceinline__ double halo_residual(const KArgs& a, const PartHalo& C, const HaloSm<V>& S, int l, double& bi) {
    bi = a.b[__ldg(&C.qa[S.p0 + l])];
    const double* val = C.val + C.ebase[blockIdx.x];
    double v = 0.0;
    for (int k = S.rp[l]; k < S.rp[l + 1]; ++k)
        v += __ldg(&val[k]) * __ldcg(&C.x[halo_global(S, (int)__ldg(&S.lcol[k]))]);
    return bi - v;
}

// FP64 CG: MODE 0 Jacobi or no preconditioner, 1 IC(0), 2 ILU(0) (pcg_part's iterations).
template <int MODE>
__device__ void pcg_halo(const KArgs& a, const PartHalo& C, double* sh, unsigned char* smem) {
    HaloSm<double> S = halo_sm<double>(C, a.A.n, smem, MODE != 0, false);
    const int tid = threadIdx.x, np = S.np;
    int* err = a.bar.err;
    int* rec = a.bar.rec;
    const bool rel = a.criterion == PF2_CRITERION_REL;
    const bool jac = a.precond == PF2_PRECOND_JACOBI;
    for (int l = tid; l < np; l += kPartThreads) __stcg(&C.x[S.p0 + l], a.x[__ldg(&C.qa[S.p0 + l])]);
    if (!grid_sync(a.bar, gridDim.x)) return;
    double red[3] = { 0.0, 0.0, 0.0 };  // r.z, b.b, r.r
    for (int l = tid; l < np; l += kPartThreads) {
        double bi;
        S.r[l] = halo_residual(a, C, S, l, bi);
        red[1] += bi * bi;
    }
    if (MODE == 0)
        for (int l = tid; l < np + S.nh; l += kPartThreads) S.t[l] = 1.0 / __ldg(&S.val[S.rp[l] + S.dg[l]]);
    __syncthreads();
    halo_publish_r(C, S);
    if (!grid_sync(a.bar, gridDim.x)) return;
    halo_fetch(C, S, S.r);
    __syncthreads();
    if (MODE == 0) {
        for (int l = tid; l < np + S.nh; l += kPartThreads) {
            const double ri = S.r[l];
            const double zi = jac ? ri * S.t[l] : ri;
            S.z[l] = zi;
            S.p[l] = zi;
            if (l < np) {
                red[0] += ri * zi;
                red[2] += ri * ri;
            }
        }
    } else {
        red[2] = halo_fwd<MODE == 1, double>(C, S, true, 0.0, true).x;
        halo_fetch_t(C, S, err, rec);
        red[0] = halo_bwd(C, S, true);
        __syncthreads();
        halo_p_update(C, S, 0.0, true);
    }
    double r2[2] = { red[0], red[1] }, r1[1] = { red[2] };
    if (!part_reduce<2>(a.bar, r2, sh, S.red)) return;
    // bnorm and the first test (thread 0; see part_reduce)
    if (!part_reduce<1>(a.bar, r1, sh, S.red, [&](const double* tot, double* out) {
            out[0] = sqrt(r2[1]);
            out[1] = rel ? (sqrt(tot[0]) <= a.tol * out[0]) : (r2[0] < a.tol * a.tol);
        }))
        return;
    double gamma = r2[0];
    const double bnorm = sh[24];
    double rr = r1[0];
    int it = 0;
    bool conv = sh[25] != 0.0;
    while (!conv && it < a.maxit) {
        ++it;
        double pq[1] = { halo_spmv(C, S) };
        if (!part_reduce<1>(a.bar, pq, sh, S.red, [&](const double* tot, double* out) { out[0] = gamma / tot[0]; }))
            return;
        const double alpha = sh[24];
        halo_fetch(C, S, S.q);
        __syncthreads();
        // with the absolute criterion (a test of r.z alone) r.r is reduced once after the loop
        double g2[2] = { 0.0, 0.0 };  // r.z (IC: t.t), r.r
        auto test = [&](const double* tot, double* out) {
            out[0] = rel ? sqrt(tot[1]) <= a.tol * bnorm : tot[0] < a.tol * a.tol;
            out[1] = tot[0] / gamma;
        };
        bool ok;
        if (MODE == 1) {
            // z = L^{-T} t does not depend on beta: the x update and the backward sweep run between
            // the arrival at the t.t (and r.r) reduction and the wait for the others
            const double2 f = halo_fwd<true, double>(C, S, false, alpha, rel);
            auto window = [&]() {
                for (int l = tid; l < np; l += kPartThreads)
                    __stcg(&C.x[S.p0 + l], __ldcg(&C.x[S.p0 + l]) + alpha * S.p[l]);
                halo_fetch_t(C, S, err, rec);
                halo_bwd(C, S, false);
            };
            if (rel) {
                double g[2] = { f.y, f.x };
                const unsigned tk = grid_reduce_tree_arrive<kPartThreads, 2>(a.bar, g, sh, S.red);
                window();
                ok = grid_reduce_tree_wait<kPartThreads, 2>(a.bar, tk, g, sh, test);
                g2[0] = g[0];
                g2[1] = g[1];
            } else {
                double g[1] = { f.y };
                const unsigned tk = grid_reduce_tree_arrive<kPartThreads, 1>(a.bar, g, sh, S.red);
                window();
                ok = grid_reduce_tree_wait<kPartThreads, 1>(a.bar, tk, g, sh, test);
                g2[0] = g[0];
            }
        } else {
            if (MODE == 0) {
                for (int l = tid; l < np + S.nh; l += kPartThreads) {
                    const double ri = S.r[l] - alpha * S.q[l];
                    const double zi = jac ? ri * S.t[l] : ri;
                    S.r[l] = ri;
                    S.z[l] = zi;
                    if (l < np) {
                        __stcg(&C.x[S.p0 + l], __ldcg(&C.x[S.p0 + l]) + alpha * S.p[l]);
                        g2[0] += ri * zi;
                        if (rel) g2[1] += ri * ri;
                    }
                }
            } else {
                g2[1] = halo_fwd<false, double>(C, S, false, alpha, rel).x;
                for (int l = tid; l < np; l += kPartThreads)
                    __stcg(&C.x[S.p0 + l], __ldcg(&C.x[S.p0 + l]) + alpha * S.p[l]);
                halo_fetch_t(C, S, err, rec);
                g2[0] = halo_bwd(C, S, true);
            }
            // the test and beta = r.z / (previous r.z) (thread 0; see part_reduce)
            if (rel) {
                ok = part_reduce<2>(a.bar, g2, sh, S.red, test);
            } else {
                double g1[1] = { g2[0] };
                ok = part_reduce<1>(a.bar, g1, sh, S.red, test);
                g2[0] = g1[0];
            }
        }
        if (!ok) return;
        if (rel) rr = g2[1];
        gamma = g2[0];
        if (sh[24] != 0.0) { conv = true; break; }
        halo_p_update(C, S, sh[25], false);
        __syncthreads();
    }
    if (!rel && it > 0) {
        double f[1] = { 0.0 };
        for (int l = tid; l < np; l += kPartThreads) f[0] += S.r[l] * S.r[l];
        if (!part_reduce<1>(a.bar, f, sh, S.red)) return;
        rr = f[0];
    }
    for (int l = tid; l < np; l += kPartThreads) a.x[__ldg(&C.qa[S.p0 + l])] = __ldcg(&C.x[S.p0 + l]);
    if (blockIdx.x == 0 && tid == 0) {
        a.out->iterations = it;
        a.out->converged = conv ? 1 : 0;
        a.out->residual = rel ? sqrt(rr) / (bnorm > 0 ? bnorm : 1.0) : sqrt(gamma);
        a.out->relres = sqrt(rr) / (bnorm > 0 ? bnorm : 1.0);
        a.out->status = conv ? DEV_OK : DEV_NOT_CONVERGED;
    }
}

// Mixed-precision CG (pcg_part_mixed's algorithm: FP32 iteration, FP64 sums, reliable updates).
template <bool IC>
__device__ void pcg_halo_mixed(const KArgs& a, const PartHalo& C, double* sh, unsigned char* smem) {
    HaloSm<float> S = halo_sm<float>(C, a.A.n, smem, true, true);
    const int tid = threadIdx.x, np = S.np;
    int* err = a.bar.err;
    int* rec = a.bar.rec;
    for (int l = tid; l < np; l += kPartThreads) {
        __stcg(&C.x[S.p0 + l], a.x[__ldg(&C.qa[S.p0 + l])]);
        S.d[l] = 0.0f;
    }
    if (!grid_sync(a.bar, gridDim.x)) return;
    // r = b - A x in FP64, published for the parts that hold it as halo
    auto residual = [&](double& rr_, double* bb_) {
        for (int l = tid; l < np; l += kPartThreads) {
            double bi;
            const double ri = halo_residual(a, C, S, l, bi);
            S.r[l] = (float)ri;
            if (S.pub[l] & 1) __stcg(&C.gq32[S.p0 + l], (float)ri);
            rr_ += ri * ri;
            if (bb_) *bb_ += bi * bi;
        }
    };
    double red[2] = { 0.0, 0.0 };  // b.b, r.r
    residual(red[1], &red[0]);
    // square roots by thread 0 (see part_reduce)
    if (!part_reduce<2>(a.bar, red, sh, S.red, [&](const double* tot, double* out) {
            out[0] = sqrt(tot[0]);
            out[1] = sqrt(tot[1]);
        }))
        return;
    const double bnorm = sh[24];
    const double target = a.tol * bnorm;
    double rnorm = sh[25];
    double rlast = rnorm;
    int it = 0, refinements = 1;
    bool conv = rnorm <= target;
    if (!conv) {
        // z = M^{-1} r, p = z, gamma = r.z
        halo_fetch(C, S, S.r);
        __syncthreads();
        halo_fwd<IC, float>(C, S, true, 0.0f, false);
        halo_fetch_t(C, S, err, rec);
        double g[1] = { halo_bwd(C, S, true) };
        __syncthreads();
        halo_p_update(C, S, 0.0f, true);
        if (!part_reduce<1>(a.bar, g, sh, S.red)) return;
        double gamma = g[0];
        while (it < a.maxit) {
            double pq[1] = { halo_spmv(C, S) };
            ++it;
            if (!part_reduce<1>(a.bar, pq, sh, S.red, [&](const double* tot, double* out) {
                    out[0] = (double)(float)(gamma / tot[0]);
                }))
                return;
            const float alpha = (float)sh[24];
            halo_fetch(C, S, S.q);
            __syncthreads();
            double g2[2];  // r.z (IC: t.t), r.r
            // refinement test and beta (thread 0; see part_reduce)
            auto post = [&](const double* tot, double* out) {
                const double rit = sqrt(tot[1]);
                out[0] = rit <= a.inner_eta * rlast || rit <= target;
                out[1] = (double)(float)(tot[0] / gamma);
            };
            const double2 f = halo_fwd<IC, float>(C, S, false, alpha, true);
            auto d_update = [&]() {
                for (int l = tid; l < np; l += kPartThreads) S.d[l] = S.d[l] + alpha * S.p[l];
            };
            g2[1] = f.x;
            if (IC) {
                // the backward sweep (z alone) overlaps the reduction, as in pcg_halo
                g2[0] = f.y;
                const unsigned tk = grid_reduce_tree_arrive<kPartThreads, 2>(a.bar, g2, sh, S.red);
                d_update();
                halo_fetch_t(C, S, err, rec);
                halo_bwd(C, S, false);
                if (!grid_reduce_tree_wait<kPartThreads, 2>(a.bar, tk, g2, sh, post)) return;
            } else {
                d_update();
                halo_fetch_t(C, S, err, rec);
                g2[0] = halo_bwd(C, S, true);
                if (!part_reduce<2>(a.bar, g2, sh, S.red, post)) return;
            }
            double gnew = g2[0];
            float beta = (float)sh[25];
            if (sh[24] != 0.0) {
                // refinement: x += d, r = b - A x and the test in FP64
                for (int l = tid; l < np; l += kPartThreads) {
                    __stcg(&C.x[S.p0 + l], __ldcg(&C.x[S.p0 + l]) + (double)S.d[l]);
                    S.d[l] = 0.0f;
                }
                if (!grid_sync(a.bar, gridDim.x)) return;
                double rr[1] = { 0.0 };
                residual(rr[0], nullptr);
                if (!part_reduce<1>(a.bar, rr, sh, S.red, [&](const double* tot, double* out) {
                        out[0] = sqrt(tot[0]);
                    }))
                    return;
                ++refinements;
                rnorm = sh[24];
                if (rnorm <= target) { conv = true; break; }
                rlast = rnorm;
                // continue from the true residual, keeping the search direction
                halo_fetch(C, S, S.r);
                __syncthreads();
                const double2 f3 = halo_fwd<IC, float>(C, S, true, 0.0f, false);
                halo_fetch_t(C, S, err, rec);
                const double rz = halo_bwd(C, S, !IC);
                double g3[1] = { IC ? f3.y : rz };
                if (!part_reduce<1>(a.bar, g3, sh, S.red, [&](const double* tot, double* out) {
                        out[0] = (double)(float)(tot[0] / gamma);
                    }))
                    return;
                gnew = g3[0];
                beta = (float)sh[24];
            }
            gamma = gnew;
            halo_p_update(C, S, beta, false);
            __syncthreads();
        }
        if (!conv)  // iteration limit: keep the accumulated update
            for (int l = tid; l < np; l += kPartThreads)
                __stcg(&C.x[S.p0 + l], __ldcg(&C.x[S.p0 + l]) + (double)S.d[l]);
    }
    for (int l = tid; l < np; l += kPartThreads) a.x[__ldg(&C.qa[S.p0 + l])] = __ldcg(&C.x[S.p0 + l]);
    if (blockIdx.x == 0 && tid == 0) {
        a.out->iterations = it;
        a.out->converged = conv ? 1 : 0;
        a.out->residual = rnorm / (bnorm > 0 ? bnorm : 1.0);
        a.out->relres = rnorm / (bnorm > 0 ? bnorm : 1.0);
        a.out->status = conv ? DEV_OK : DEV_NOT_CONVERGED;
        a.out->pad = refinements;
    }
}

template <int MODE>
__global__ void __launch_bounds__(kPartThreads, 1) k_pcg_halo(KArgs a, PartHalo C) {
    __shared__ double sh[kShDoubles];
    extern __shared__ __align__(16) unsigned char part_smem[];
    pcg_halo<MODE>(a, C, sh, part_smem);
}

template <bool IC>
__global__ void __launch_bounds__(kPartThreads, 1) k_pcg_halo_mixed(KArgs a, PartHalo C) {
    __shared__ double sh[kShDoubles];
    extern __shared__ __align__(16) unsigned char part_smem[];
    pcg_halo_mixed<IC>(a, C, sh, part_smem);
}

}  // namespace pf2

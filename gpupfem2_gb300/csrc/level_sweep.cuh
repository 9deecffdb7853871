// level_sweep.cuh - CG with ILU(0)/IC(0) in the natural order of a mesh, whose triangular solves
// are chains of many levels; included by solvers.cu.
//
// A level of a few dozen rows costs its latency: 1.6 us where values go between SMs through L2.
// Here one block solves the triangles, with the solved values in shared memory, and the other
// blocks share the SpMV and the vector updates.
//
// Rows take slots in level order, in slices of 32 and units of at most kLevelSlices slices; a
// level with more rows is several units (which then also count as levels below).  Solved values go
// to a shared-memory ring of the last kLevelRing slots; the rare dependency older than that is
// read from where the sweep writes its results.  Four groups of four warps (a warp of each SM
// sub-partition) take the units in turn, in three steps between block barriers:
//   l - 3  the group that has just finished unit l - 4 issues the loads of unit l, coalesced from
//          L2 into registers: right-hand side (kept in slot order), inverse pivots, factor values
//          and ring positions;
//   l      it sums the dependencies that lie before unit l - 1 ("early");
//   l + 1  it adds those in unit l - 1 ("late": their factors are already scaled by the inverse
//          pivot) and stores the results.
// So between two barriers there are only one read of the ring, the late products and the store.
//
// What bounds it: the chain.  16,705 rows (257 x 65 nodes, 321 levels of ~52 rows): 160 us per
// ILU(0) iteration, 1,046 with the banded solve; a unit takes ~440 clocks, of which the barrier
// 43, the ring 30 and two late products 128 (64 clocks per FP64 warp instruction); on wide meshes
// the FP64 pipe.  Before the three steps were split: 449 (units through a
// bulk-copy ring, two groups; its mbarriers cost ~300 clocks a unit), 328 (loads issued beside the
// late products), 212 (the generic sums on the path of the common ones).
#pragma once

namespace pf2 {

constexpr int kLevelRing = 16384;   // slots of the ring (128 KB)
constexpr int kLevelSlices = 4;     // slices of a unit: the warps of a group
constexpr int kLevelGroups = 4;
constexpr int kLevelThreads = 32 * kLevelSlices * kLevelGroups;
constexpr int kLevelCase = 8;       // early and late dependencies of a row kept in registers
constexpr int kLevelFar = 1 << 24;  // LevelSweep::unit flag: some dependencies have left the ring
constexpr int kLevelSmem = 8 * kLevelRing;

struct LevelSweep {
    const unsigned char* stream;
    const int4* unit;  // offset / 16 in stream; early dependencies | late << 8 | slices << 16 | flags; first slot
    int units;         // a multiple of kLevelGroups (the last ones empty)
};

struct LevelCg {
    LevelSweep f, b;
    const int* slot_f;  // row -> forward slot
    double* rf;         // right-hand side of the forward sweep by forward slot
    double* tb;         // forward result by backward slot
};

// A slice with K dependencies: inverse pivots (32 x 8 bytes), ring positions, destinations (32 x 4
// each), then K times factor values and the positions of the values they multiply (in the ring,
// bytes; ~destination for one that has left it).
__host__ __device__ constexpr int level_slice_bytes(int K) { return 512 + 384 * K; }

// s - sum of the K dependencies (factors f, positions d) in the ring.
template <int K>
__device__ __forceinline__ double level_sub(double s, const double* f, const int* d, const unsigned char* ring) {
    double v[K + 1];
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = *reinterpret_cast<const double*>(ring + d[k]);
#pragma unroll
    for (int k = 0; k < K; ++k) s = __fma_rn(-f[k], v[k], s);
    return s;
}

// One sweep by all threads of a block: ring and out[destination] = result.  in: right-hand side by
// slot.  pivot: rows are divided by their pivot.
__device__ __forceinline__ void level_sweep(const LevelSweep& S, const double* in, double* out, bool pivot,
                                            unsigned char* ring) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, g = w / kLevelSlices;
    // consecutive narrow units use different sub-partitions
    const int sl = (w + 2 * g) % kLevelSlices;
    double s = 0.0, piv = 1.0, ev[kLevelCase], lv[kLevelCase];
    int ei[kLevelCase], li[kLevelCase], early = 0, late = 0, pos = 0, dest = -1;
    const unsigned char* more = nullptr;  // early dependencies beyond kLevelCase
    // how to sum: the number of dependencies, 0 .. kLevelCase, all in the ring; kNone: the warp has
    // no slice of the unit; kAny: else (a branch to code for exactly that number: a predicated-off
    // FP64 instruction still takes the pipe's 64 clocks, and so do the jumps of a longer test)
    constexpr int kNone = -1, kAny = kLevelCase + 1;
    int sum_early = kNone, sum_late = kNone;
    auto unit_at = [&](int l) { return l < S.units ? __ldg(&S.unit[l]) : make_int4(0, 0, 0, 0); };
    auto value_far = [&](int d) {
        return d >= 0 ? *reinterpret_cast<const double*>(ring + d) : __ldcg(&out[~d]);
    };
    auto load = [&](int4 u) {
        asm volatile("" : "+r"(u.x), "+r"(u.y), "+r"(u.z));  // (not waited for where it is loaded)
        sum_early = sum_late = kNone;
        if (sl >= ((u.y >> 16) & 15)) return;
        early = u.y & 255;
        late = (u.y >> 8) & 255;
        sum_early = u.y & kLevelFar ? kAny : min(early, kAny);
        sum_late = u.y & kLevelFar ? kAny : late;
        const unsigned char* p = S.stream + 16ll * u.x + sl * level_slice_bytes(early + late);
        const unsigned char *pd = p + 8 * lane, *pi = p + 4 * lane;
        s = __ldcg(&in[u.z + 32 * sl + lane]);
        piv = __ldg(reinterpret_cast<const double*>(pd));
        pos = __ldg(reinterpret_cast<const int*>(pi + 256));
        dest = __ldg(reinterpret_cast<const int*>(pi + 384));
#pragma unroll
        for (int k = 0; k < kLevelCase; ++k)
            if (k < early) {
                ev[k] = __ldg(reinterpret_cast<const double*>(pd + 512 + 384 * k));
                ei[k] = __ldg(reinterpret_cast<const int*>(pi + 768 + 384 * k));
            }
        more = p + 512 + 384 * kLevelCase;
        pd += 384 * early;
        pi += 384 * early;
#pragma unroll
        for (int k = 0; k < kLevelCase; ++k)
            if (k < late) {
                lv[k] = __ldg(reinterpret_cast<const double*>(pd + 512 + 384 * k));
                li[k] = __ldg(reinterpret_cast<const int*>(pi + 768 + 384 * k));
            }
    };
    auto sub = [&](int how, int count, const double* f, const int* d) {
        switch (how) {
            case 0: break;
            case 1: s = level_sub<1>(s, f, d, ring); break;
            case 2: s = level_sub<2>(s, f, d, ring); break;
            case 3: s = level_sub<3>(s, f, d, ring); break;
            case 4: s = level_sub<4>(s, f, d, ring); break;
            case 5: s = level_sub<5>(s, f, d, ring); break;
            case 6: s = level_sub<6>(s, f, d, ring); break;
            case 7: s = level_sub<7>(s, f, d, ring); break;
            case 8: s = level_sub<8>(s, f, d, ring); break;
            default:
#pragma unroll
                for (int k = 0; k < kLevelCase; ++k)
                    if (k < count) s = __fma_rn(-f[k], value_far(d[k]), s);
        }
    };
    for (int i = 0; i < g; ++i) __syncthreads();
    load(unit_at(g));
    int4 next = unit_at(g + kLevelGroups);
    for (int l = g; l < S.units; l += kLevelGroups) {
        __syncthreads();  // unit l - 2 is solved
        if (sum_early != kNone) {
            if (__builtin_expect(sum_early == 1, 1)) s = level_sub<1>(s, ev, ei, ring);
            else sub(sum_early, early, ev, ei);
            for (int k = kLevelCase; k < early; ++k, more += 384)
                s = __fma_rn(-__ldg(reinterpret_cast<const double*>(more) + lane),
                             value_far(__ldg(reinterpret_cast<const int*>(more + 256) + lane)), s);
            if (pivot) s *= piv;
        }
        __syncthreads();  // unit l - 1 is solved
        if (__builtin_expect(sum_late == 2, 1)) {
            s = level_sub<2>(s, lv, li, ring);
            *reinterpret_cast<double*>(ring + pos) = s;
            if (dest >= 0) __stcg(&out[dest], s);
        } else if (sum_late != kNone) {
            sub(sum_late, late, lv, li);
            *reinterpret_cast<double*>(ring + pos) = s;
            if (dest >= 0) __stcg(&out[dest], s);
        }
        __syncthreads();
        load(next);
        next = unit_at(l + 2 * kLevelGroups);
        __syncthreads();
    }
    for (int i = g; i < kLevelGroups; ++i) __syncthreads();
}

// z = M^{-1} r, by one block.
__global__ void __launch_bounds__(kLevelThreads, 1) k_level_apply(KArgs a, LevelCg C) {
    extern __shared__ __align__(128) unsigned char level_ring[];
    for (int i = threadIdx.x; i < a.A.n; i += blockDim.x) __stcg(&C.rf[__ldg(&C.slot_f[i])], a.r[i]);
    __syncthreads();
#pragma unroll 1
    for (int d = 0; d < 2; ++d)
        level_sweep(d ? C.b : C.f, d ? C.tb : C.rf, d ? a.z : C.tb, d || a.precond == PF2_PRECOND_IC, level_ring);
}

// SolverCG::solve with ILU(0)/IC(0), k_pcg's iteration: q = A p with p.q; x, r; z = M^{-1} r by
// block 0; r.z and r.r; p.
__global__ void __launch_bounds__(kLevelThreads, 1) k_pcg_level(KArgs a, LevelCg C) {
    __shared__ double sh[kShDoubles];
    extern __shared__ __align__(128) unsigned char level_ring[];
    const bool rel = a.criterion == PF2_CRITERION_REL;
    const bool ic = a.precond == PF2_PRECOND_IC;
    int r0, r1;
    row_range(a.A.n, r0, r1);
    // r = b - A x
    for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
        const double ri = a.b[i] - row_dot(a.A, i, a.x);
        a.r[i] = ri;
        __stcg(&C.rf[__ldg(&C.slot_f[i])], ri);
    }
    auto precondition = [&]() {
        if (!grid_sync(a.bar, gridDim.x)) return false;
        if (blockIdx.x == 0) {
#pragma unroll 1
            for (int d = 0; d < 2; ++d)
                level_sweep(d ? C.b : C.f, d ? C.tb : C.rf, d ? a.z : C.tb, d || ic, level_ring);
        }
        return grid_sync(a.bar, gridDim.x);
    };
    if (!precondition()) return;
    double red[3] = { 0.0, 0.0, 0.0 };  // r.z, b.b, r.r
    for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
        const double zi = __ldcg(&a.z[i]), ri = a.r[i], bi = a.b[i];
        __stcg(&a.p[i], zi);
        red[0] += ri * zi;
        red[1] += bi * bi;
        red[2] += ri * ri;
    }
    if (!grid_reduce<3>(a.bar, red, sh)) return;
    double gamma = red[0], rr = red[2];
    const double bnorm = sqrt(red[1]), tol2 = a.tol * a.tol;
    auto done = [&]() { return rel ? sqrt(rr) <= a.tol * bnorm : gamma < tol2; };
    int it = 0;
    bool conv = done();
    while (!conv && it < a.maxit) {
        ++it;
        double pq[1] = { spmv_rows(a.A, a.p, a.q, r0, r1) };
        if (!grid_reduce<1>(a.bar, pq, sh)) return;
        const double alpha = gamma / pq[0];
        double g2[2] = { 0.0, 0.0 };  // r.z, r.r
        for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
            a.x[i] += alpha * a.p[i];
            const double ri = a.r[i] - alpha * a.q[i];
            a.r[i] = ri;
            __stcg(&C.rf[__ldg(&C.slot_f[i])], ri);
            g2[1] += ri * ri;
        }
        if (!precondition()) return;
        for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) g2[0] += a.r[i] * __ldcg(&a.z[i]);
        if (!grid_reduce<2>(a.bar, g2, sh)) return;
        rr = g2[1];
        const double beta = g2[0] / gamma;
        gamma = g2[0];
        if (done()) {
            conv = true;
            break;
        }
        p_update(a.p, a.z, beta, r0, r1);
        if (!grid_sync(a.bar, gridDim.x)) return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out->iterations = it;
        a.out->converged = conv ? 1 : 0;
        a.out->residual = rel ? sqrt(rr) / (bnorm > 0 ? bnorm : 1.0) : sqrt(gamma);
        a.out->relres = sqrt(rr) / (bnorm > 0 ? bnorm : 1.0);
        a.out->status = conv ? DEV_OK : DEV_NOT_CONVERGED;
    }
}

}  // namespace pf2

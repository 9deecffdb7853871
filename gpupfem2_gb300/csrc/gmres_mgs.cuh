// gmres_mgs.cuh - GMRES with modified Gram-Schmidt in two grid-wide steps per iteration,
// included by solvers.cu.
//
// SolverGMRES::solve (linear_solver.cu:560-660) projects the new vector w on v_0, v_1, ... one
// after another, one grid-wide reduction each: (k + 1) of them in iteration k, ~2.5 us apiece.
// The same coefficients are h_i = v_i.w - sum_{j < i} (v_i.v_j) h_j, that is h = (I + L)^{-1} V^T w
// with L the strictly lower part of V^T V (the inverse compact WY form of modified Gram-Schmidt:
// Swirydowicz, Langou, Ananthan, Yang, Thomas, "Low synchronization Gram-Schmidt and generalized
// minimal residual algorithms", 2021), with modified Gram-Schmidt's loss of orthogonality.  An
// iteration takes V^T w and the new row V^T v_k of L in one pass over V and one exchange, solves
// for h, updates w, and reduces its norm.
//
// The exchange: block b sends its parts of the 2 k + 1 sums as packets (value and exchange number
// in one word, part_halo.cuh), block i mod G adds up value i in block order and sends the total to
// all.  w before its normalisation is what the next product reads (times 1 / ||w||), so the
// normalised rows need no grid-wide step of their own; the Givens rotations of a column run in
// one warp beside that product, whose last one is thrown away.
//
// What bounds it: FP64 issue for large systems (3 multiply-adds per entry of V, 64 clocks per warp
// instruction on a sub-partition: 25,000 of 63,000 clocks an iteration at 125,364 rows and a mean
// basis of 17), the latency of its dependent steps for small ones.  Velocity prediction with
// Jacobi, one reduction per projection -> this: 125,364 rows, 34 iterations, 4.69 -> 1.14 ms;
// 16,705 rows, 23 iterations, 0.40 ms.  One block per SM (128 registers a thread) against two:
// 1.13 / 1.49 ms at 125,364 rows, 9.5 / 9.3 at 499,288 (v_k scaled, not divided); 128 rows a block at least against 512:
// 0.40 / 0.59 ms at 16,705 rows.  Norms by packets and a fence against grid_reduce: 8,600 against
// 11,500 clocks.
#pragma once

namespace pf2 {

struct GmresMgs {
    // (the rows of L, written by block 0, lie in H's unused triangle: v_i.v_j, j < i, at m j + i)
    unsigned long long* part;  // packets (zeroed before the launch): 2 x (2 m + 2) x G parts, 2 x (2 m + 2)
                               // totals, 2 x G parts of norms; then the counter of norm parts
};

__host__ __device__ constexpr size_t gmres_packet_words(int m, int G) {
    return 2 * 2 * ((size_t)(2 * m + 2) * (G + 1) + G) + 2;
}

constexpr int kGramRows = 96;                                            // rows of L that each block keeps
constexpr size_t kGramBytes = sizeof(double) * (kGramRows + 1) * (kGramRows + 1);  // (dynamic shared memory)
constexpr int kGmresRows = 128;                                          // rows per block at least
// Rows per block from which on the basis no longer stays in L2 and a block's loads in flight set
// the pace: rows then go four (product) and two (update) at a time, and all 16 warps take part in
// the dot products of a short basis.  1,997,113 rows, Jacobi, ms per solve, one reduction per projection
// with two blocks per SM / without this / with it: 8 iterations 1.52 / 1.70 / 1.53, 40 iterations
// 17.3 / 15.9 / 13.3, 40 restarted after 10 7.96 / 8.88 / 7.67.  Below, the loads cost more than they
// hide: 125,364 rows, 40 iterations 1.34 without, 1.45 with.
constexpr int kGmresMany = 4096;

// f(i, (A x)_i) for rows i0, i0 + step, .. below r1, N of them with their loads in flight together
// (each row's entries in order, as row_dot).
template <int N, class F>
__device__ __forceinline__ void gmres_rows(const Csr& A, const double* x, int i0, int step, int r1, F f) {
    int s[N], e[N], len = 0;
    double sum[N];
#pragma unroll
    for (int u = 0; u < N; ++u) {
        const int i = i0 + u * step;
        s[u] = i < r1 ? __ldg(&A.rowptr[i]) : 0;
        e[u] = i < r1 ? __ldg(&A.rowptr[i + 1]) : 0;
        sum[u] = 0.0;
        len = max(len, e[u] - s[u]);
    }
    for (int k = 0; k < len; ++k)
#pragma unroll
        for (int u = 0; u < N; ++u)
            if (s[u] + k < e[u]) sum[u] += __ldg(&A.val[s[u] + k]) * __ldcg(&x[__ldg(&A.col[s[u] + k])]);
#pragma unroll
    for (int u = 0; u < N; ++u)
        if (i0 + u * step < r1) f(i0 + u * step, sum[u]);
}

// Sums over this block's rows j = lo + lane, ... of w V_i and u V_i for C vectors i: lane 4 q's
// low bits zero, bits 2..4 = q: value q (w V_0, ..; from C on u V_0, ..).
template <int C>
__device__ __forceinline__ double gmres_dots(const double* V, size_t n, const double* w, const double* u, int lo, int hi) {
    const int lane = threadIdx.x & 31;
    double d[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) d[q] = 0.0;
#pragma unroll 2
    for (int j = lo + lane; j < hi; j += 32) {
        const double wj = w[j], uj = u[j];
        double v[C];
#pragma unroll
        for (int q = 0; q < C; ++q) v[q] = V[q * n + j];
#pragma unroll
        for (int q = 0; q < C; ++q) {
            d[q] += wj * v[q];
            d[4 + q] += uj * v[q];
        }
    }
    // each step adds two lanes' halves of the values left
#pragma unroll
    for (int s = 4; s >= 1; s /= 2) {
        const int x = 4 * s;  // lane distance 16, 8, 4
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (q < s) {
                const bool up = lane & x;
                const double give = up ? d[q] : d[q + s], keep = up ? d[q + s] : d[q];
                d[q] = keep + __shfl_xor_sync(0xffffffffu, give, x);
            }
    }
    d[0] += __shfl_xor_sync(0xffffffffu, d[0], 2);
    d[0] += __shfl_xor_sync(0xffffffffu, d[0], 1);
    return d[0];
}

// h <- (I + L)^{-1} h, rows 0 .. k; row i of L is in shared memory (Ls, leading dimension
// kGramRows + 1) below kGramRows, else in L, row k in g.  All threads of the block.
__device__ __forceinline__ void gmres_solve_lower(double* h, const double* g, const double* Ls, const double* L, int ld,
                                                  int k) {
    const int lane = threadIdx.x & 31;
    auto entry = [&](int i, int j) {
        return i < kGramRows ? Ls[j * (kGramRows + 1) + i] : i == k ? g[j] : __ldcg(&L[(size_t)j * ld + i]);
    };
    for (int base = 0; base <= k; base += 32) {
        const int nb = min(32, k + 1 - base);
        if (threadIdx.x < 32) {
            const int i = min(base + lane, k);
            double hi = h[i];
            if (k < kGramRows) {  // (what lies on and above the diagonal is read and not used)
                const double* col = Ls + base * (kGramRows + 1) + i;
                double l = *col;
#pragma unroll 1
                for (int e = 0; e < nb; ++e) {
                    const double f = lane > e ? l : 0.0;
                    col += kGramRows + 1;
                    l = *col;
                    hi -= f * __shfl_sync(0xffffffffu, hi, e);
                }
            } else {
#pragma unroll 1
                for (int e = 0; e < nb; ++e) {
                    const double f = base + e < i ? entry(i, base + e) : 0.0;
                    hi -= f * __shfl_sync(0xffffffffu, hi, e);
                }
            }
            if (lane < nb) h[i] = hi;
        }
        __syncthreads();
        if (base + 32 > k) break;
        for (int i = base + 32 + threadIdx.x; i <= k; i += blockDim.x) {
            double s = h[i];
#pragma unroll 8
            for (int e = 0; e < 32; ++e) s -= entry(i, base + e) * h[base + e];
            h[i] = s;
        }
        __syncthreads();
    }
}

// Givens rotations of column c (h[0 .. c], norm aux below it) by one warp; the rotated column goes
// to h, beta[c], beta[c + 1] follow (updateHcolumn, linear_solver.cu:40-66).
__device__ __forceinline__ void gmres_rotate(double* h, double* cs, double* sn, double* beta, int c, double aux) {
    const int lane = threadIdx.x & 31;
    double t = h[0];  // the entry that the next rotation mixes, in every lane
    for (int base = 0; base < c; base += 32) {
        const int nb = min(32, c - base), i = base + lane;
        double ci = 0.0, si = 0.0, hn = 0.0, mine = 0.0;
        if (lane < nb) {
            ci = cs[i];
            si = sn[i];
            hn = h[i + 1];
        }
        const double q = ci * hn;
        for (int e = 0; e < nb; ++e) {
            if (lane == e) mine = t;
            t = __shfl_sync(0xffffffffu, q, e) - __shfl_sync(0xffffffffu, si, e) * t;
        }
        __syncwarp();
        if (lane < nb) h[i] = ci * mine + si * hn;
        __syncwarp();
    }
    if (lane == 0) {
        const double coeff = rsqrt(t * t + aux * aux);
        cs[c] = t * coeff;
        sn[c] = aux * coeff;
        h[c] = cs[c] * t + sn[c] * aux;
        beta[c + 1] = -sn[c] * beta[c];
        beta[c] *= cs[c];
    }
    __syncwarp();
}

// y (in s on return) from the k x k upper triangle H (leading dimension m) and s, by one warp; inv
// takes the inverse diagonal.
__device__ __forceinline__ void gmres_solve_upper(double* s, double* inv, const double* H, int m, int k) {
    const int lane = threadIdx.x & 31;
    for (int i = lane; i < k; i += 32) inv[i] = 1.0 / __ldcg(&H[i + (size_t)m * i]);
    __syncwarp();
    auto entry = [&](int i, int j) { return i < j ? __ldcg(&H[i + (size_t)m * j]) : 0.0; };
    double next = entry(lane, k - 1);
    for (int j = k - 1; j >= 0; --j) {
        const double first = next, y = s[j] * inv[j];
        if (j > 0) next = entry(lane, j - 1);
        __syncwarp();
        if (lane < j) s[lane] -= first * y;
        for (int i = lane + 32; i < j; i += 32) s[i] -= entry(i, j) * y;
        if (lane == 0) s[j] = y;
        __syncwarp();
    }
}

// MANY: kGmresMany rows per block and more.
template <bool MANY>
__global__ void __launch_bounds__(kSolverThreads, 1) k_gmres_mgs(KArgs a, GmresMgs C) {
    const int ep_base = a.epoch ? *a.epoch : 0;  // read before the counter can advance
    __shared__ double sh[kShDoubles];  // (grid_sync, norm)
    __shared__ double cs[kMaxGmresSmem], sn[kMaxGmresSmem], beta[kMaxGmresSmem + 1], h[kMaxGmresSmem + 1];
    __shared__ double g[kMaxGmresSmem + 1];
    __shared__ double red[kSolverThreads];
    constexpr int kWarps = kSolverThreads / 32;
    double* const seg_sum = red;
    double* const Ls = reinterpret_cast<double*>(pf2_band_smem) + (a.T.band.P ? a.T.band.R : 0);
    int r0, r1;
    row_range(a.A.n, r0, r1);
    const int n = a.A.n, m = a.m, G = (int)gridDim.x;
    const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
    const int nval = 2 * m + 2;
    unsigned long long* const tot = C.part + 2 * 2 * (size_t)nval * G;
    const bool global_pc = (a.precond == PF2_PRECOND_ILU || a.precond == PF2_PRECOND_IC);
    if (a.precond == PF2_PRECOND_JACOBI)
        for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) a.invd[i] = 1.0 / a.A.val[a.A.diag[i]];
    const bool jacobi = a.precond == PF2_PRECOND_JACOBI;
    double* const raw = a.z;  // the newest vector before its normalisation, read by other blocks
    double* const w = a.p;    // own rows
    int apply = 0, total_it = 0;
    bool conv = false;
    double res = 0.0;
    unsigned seq = 0, norms = 0;
    unsigned long long* const norm_part = tot + 2 * 2 * (size_t)nval;
    unsigned* const norm_count = reinterpret_cast<unsigned*>(norm_part + 2 * 2 * (size_t)G);
    // sqrt of the grid-wide sum of v; all blocks' earlier stores are visible behind it.  False on
    // a timeout or an error.
    auto norm = [&](double v, double& result) {
        red[threadIdx.x] = v;
        __syncthreads();
        if (threadIdx.x < 64) {
            double t = red[threadIdx.x];
#pragma unroll
            for (int e = 1; e < kSolverThreads / 64; ++e) t += red[threadIdx.x + 64 * e];
            red[threadIdx.x] = t;
        }
        __syncthreads();
        ++norms;
        unsigned long long* const mine = norm_part + 2 * (size_t)(norms & 1) * G;
        int ok = 1;
        if (wq == 0) {
            if (lane == 0) __threadfence();  // the block's stores, before its part
            double t = warp_sum(red[lane] + red[lane + 32]);
            if (lane == 0) {
                HaloPacket<double>::put(mine + 2 * (size_t)blockIdx.x, t, norms);
                asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" : : "l"(norm_count) : "memory");
            }
            if (lane == 0 && G >= (int)kHaloCountBlocks) {
                const unsigned target = norms * (unsigned)G;
                long long polls = 0;
                while ((int)(ld_relaxed_gpu(norm_count) - target) < 0) {
                    if (++polls > (a.bar.max_polls > 0 ? a.bar.max_polls : kBarrierPolls)) {
                        atomicExch(a.bar.err, (int)DEV_TIMEOUT);
                        record_timeout(a.bar.rec, 1, (int)blockIdx.x, (int)norms, 0, 0);
                        break;
                    }
                    if ((polls & 255) == 0 && *(volatile int*)a.bar.err != 0) break;
                }
            }
            __syncwarp();
            t = 0.0;
            for (int q0 = lane; q0 < G; q0 += 5 * 32) {
                double x[5];
                bool here[5];
#pragma unroll
                for (int e = 0; e < 5; ++e)
                    here[e] = q0 + 32 * e < G && HaloPacket<double>::get(mine + 2 * (size_t)(q0 + 32 * e), x[e], norms);
#pragma unroll
                for (int e = 0; e < 5; ++e)
                    if (q0 + 32 * e < G)
                        t += halo_settle<double>(mine + 2 * (size_t)(q0 + 32 * e), here[e], x[e], norms, a.bar, 1, 0);
            }
            t = warp_sum(t);
            __threadfence();  // the others' stores, behind their parts
            if (lane == 0) {
                sh[0] = sqrt(t);
                ok = *(volatile int*)a.bar.err == 0;
            }
        }
        ok = __syncthreads_and(ok);
        result = sh[0];
        return ok != 0;
    };
    while (true) {
        // v0 = M^{-1}(b - A x), beta0 = ||v0||
        for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) a.r[i] = a.b[i] - row_dot(a.A, i, a.x);
        __syncthreads();
        if (global_pc && !grid_sync(a.bar, gridDim.x)) return;
        if (!precond_apply(a, a.r, w, r0, r1, apply++, ep_base)) return;
        __syncthreads();
        double nn = 0.0, aux;
        for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
            const double v = w[i];
            __stcg(&raw[i], v);
            nn += v * v;
        }
        if (!norm(nn, aux)) return;
        res = aux;
        if (res < a.tol) { conv = true; break; }
        if (total_it >= a.maxit) break;
        if (threadIdx.x == 0) beta[0] = aux;
        int k = 0;
        bool inner_conv = false;
        while (true) {
            // v_k (own rows) and w = M^{-1} A v_k; the last column's rotations by warp 0
            const double inv = 1.0 / aux;
            double* vk = a.V + (size_t)k * n;
            double* out = global_pc ? a.q : w;
            if (k > 0 && wq == 0) {
                gmres_rotate(h, cs, sn, beta, k - 1, aux);
                if (blockIdx.x == 0)
                    for (int i = lane; i < k; i += 32) __stcg(&a.H[(size_t)m * (k - 1) + i], h[i]);
            } else {
                const int skip = k > 0 ? 32 : 0;
                const int step = (int)blockDim.x - skip;
                auto put = [&](int i, double sum) {
                    vk[i] = __ldcg(&raw[i]) / aux;
                    const double v = sum * inv;
                    out[i] = jacobi ? v * a.invd[i] : v;
                };
                if constexpr (MANY)
                    for (int i = r0 + threadIdx.x - skip; i < r1; i += 4 * step) gmres_rows<4>(a.A, raw, i, step, r1, put);
                else
                    for (int i = r0 + threadIdx.x - skip; i < r1; i += step) put(i, row_dot(a.A, i, raw));
            }
            __syncthreads();
            if (k > 0) res = fabs(beta[k]);
            if (k > 0 && res < a.tol) { inner_conv = true; break; }
            if (k == m || total_it >= a.maxit) break;
            ++total_it;
            if (global_pc) {
                if (!grid_sync(a.bar, gridDim.x)) return;
                if (!precond_apply(a, a.q, w, r0, r1, apply++, ep_base)) return;
                __syncthreads();
            }
            // V^T w and V^T v_k: tasks of four vectors and a segment of the rows, eight of them at least (many rows: 16)
            const unsigned s = ++seq;
            unsigned long long* const part = C.part + 2 * (size_t)(s & 1) * nval * G;
            unsigned long long* const total = tot + 2 * (size_t)(s & 1) * nval;
            const int groups = (k + 4) / 4, segs = max(1, (MANY ? 16 : 8) / groups), len = (r1 - r0 + segs - 1) / segs;
            // value of vector i: i (w) or k + 1 + i (v_k; none for i = k)
            auto send = [&](int i, int which, double v) {
                if (which ? i < k : i <= k)
                    HaloPacket<double>::put(part + 2 * ((size_t)(which * (k + 1) + i) * G + blockIdx.x), v, s);
            };
            for (int t = wq; t < groups * segs; t += kWarps) {
                const int gr = t / segs, seg = t % segs, lo = r0 + seg * len, hi = min(r1, lo + len);
                const double* V = a.V + (size_t)(4 * gr) * n;
                double d;
                switch (min(4, k + 1 - 4 * gr)) {
                    case 1: d = gmres_dots<1>(V, n, w, vk, lo, hi); break;
                    case 2: d = gmres_dots<2>(V, n, w, vk, lo, hi); break;
                    case 3: d = gmres_dots<3>(V, n, w, vk, lo, hi); break;
                    default: d = gmres_dots<4>(V, n, w, vk, lo, hi);
                }
                if (lane % 4 == 0) {
                    const int q = lane / 4;
                    if (segs == 1) send(4 * gr + q % 4, q / 4, d);
                    else seg_sum[8 * t + q] = d;
                }
            }
            if (segs > 1) {
                __syncthreads();
                for (int v = threadIdx.x; v < 8 * groups; v += blockDim.x) {
                    const int gr = v / 8, q = v % 8;
                    double d = 0.0;
                    for (int e = 0; e < segs; ++e) d += seg_sum[8 * (gr * segs + e) + q];
                    send(4 * gr + q % 4, q / 4, d);
                }
            }
            if (wq == 0) {  // this block's totals
                for (int v = blockIdx.x; v < 2 * k + 1; v += G) {
                    double d = 0.0;
                    for (int q0 = lane; q0 < G; q0 += 8 * 32) {  // eight loads in flight
                        double x[8];
                        bool here[8];
                        const unsigned long long* p = part + 2 * ((size_t)v * G + q0);
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            here[e] = q0 + 32 * e < G && HaloPacket<double>::get(p + 64 * e, x[e], s);
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            if (q0 + 32 * e < G) d += halo_settle<double>(p + 64 * e, here[e], x[e], s, a.bar, 1, 0);
                    }
                    d = warp_sum(d);
                    if (lane == 0) HaloPacket<double>::put(total + 2 * (size_t)v, d, s);
                }
            } else {
                for (int v = threadIdx.x - 32; v < 2 * k + 1; v += blockDim.x - 32) {
                    const double d = halo_settle<double>(total + 2 * (size_t)v, false, 0.0, s, a.bar, 1, 0);
                    if (v <= k) {
                        h[v] = d;
                    } else {
                        g[v - k - 1] = d;
                        if (k < kGramRows) Ls[(v - k - 1) * (kGramRows + 1) + k] = d;
                        if (blockIdx.x == 0) __stcg(&a.H[(size_t)(v - k - 1) * m + k], d);
                    }
                }
            }
            __syncthreads();
            gmres_solve_lower(h, g, Ls, a.H, m, k);
            nn = 0.0;
            if constexpr (MANY) {  // two rows of a thread together
                for (int j = r0 + threadIdx.x; j < r1; j += 2 * blockDim.x) {
                    const bool two = j + (int)blockDim.x < r1;
                    const int j2 = two ? j + (int)blockDim.x : j;
                    double v = w[j], v2 = w[j2];
#pragma unroll 4
                    for (int i = 0; i <= k; ++i) {
                        const double* Vi = a.V + (size_t)i * n;
                        v -= h[i] * Vi[j];
                        v2 -= h[i] * Vi[j2];
                    }
                    __stcg(&raw[j], v);
                    nn += v * v;
                    if (two) {
                        __stcg(&raw[j2], v2);
                        nn += v2 * v2;
                    }
                }
            } else {
                for (int j = r0 + threadIdx.x; j < r1; j += blockDim.x) {
                    double v = w[j];
#pragma unroll 4
                    for (int i = 0; i <= k; ++i) v -= h[i] * a.V[(size_t)i * n + j];
                    __stcg(&raw[j], v);
                    nn += v * v;
                }
            }
            if (!norm(nn, aux)) return;
            ++k;
        }
        // y = H^{-1} beta (upper triangular), x += V y (own rows)
        if (!grid_sync(a.bar, gridDim.x)) return;  // H's last column
        for (int i = threadIdx.x; i < k; i += blockDim.x) h[i] = beta[i];
        __syncthreads();
        if (wq == 0) gmres_solve_upper(h, g, a.H, m, k);
        __syncthreads();
        const bool update = inner_conv || (k == m && m < a.maxit);
        if (update)
            for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
                double s = 0.0;
                for (int j = 0; j < k; ++j) s += a.V[(size_t)j * n + i] * h[j];
                a.x[i] = s + a.x[i];
            }
        if (!grid_sync(a.bar, gridDim.x)) return;
        if (inner_conv) { conv = true; break; }
        if (!update || total_it >= a.maxit) break;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out->iterations = total_it;
        a.out->converged = conv ? 1 : 0;
        a.out->residual = res;
        a.out->relres = 0.0;  // GMRES tracks the preconditioned residual only
        a.out->status = conv ? DEV_OK : DEV_NOT_CONVERGED;
    }
}

}  // namespace pf2

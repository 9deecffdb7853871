// part_halo.cuh - partitioned CG with halo rows (included by solvers.cu).
//
// k_pcg_part's sweeps wait, colour by colour, for other parts' boundary values, and a third
// grid-wide step per iteration publishes the boundary rows' direction.  Here each part also
// computes the few rows around it that its own rows depend on (the same arithmetic on the same
// inputs, so the same bits as their owner), and an iteration has no wait inside a sweep:
//   F rows: other parts' rows that the part's forward sweep reads, closed under the sweep's
//           dependencies (lower groups).  Their r lives here too: r -= alpha q with the owner's
//           q, which owners publish before the p.q reduction and which is read beside it.
//   Z rows: the neighbour rows of the part's rows (ring 1, whose p the SpMV reads), closed under
//           the backward sweep's dependencies (higher groups).  Their forward result t is either
//           computed here (F rows) or read once from the owner.
// p on ring 1 follows from its z, so the direction needs no exchange.  Per iteration: SpMV;
// reduction of p.q; forward sweep; (IC(0): arrival at the t.t reduction;) t of the Z rows that
// are not F rows; backward sweep; reduction (IC(0): the wait alone).
//
// Local numbering of part k: its rows 0 .. np - 1 (Q order), then its halo rows by group, each
// group's rows as F only, F and Z, Z only.  Columns are local (16 bits), so no lookup or branch
// tells own entries from others'.
//
// Rows are taken in slices of 32 by warps (slice i of the SpMV, and of each group of a sweep, by
// warp i mod kHaloWarps).  A slice's entries, entry k of its rows side by side, lie in items of
// at most kHaloItem entry rows, and a warp's items lie in the order in which it uses them (forward
// sweep, backward sweep, SpMV).  A sweep slice's first entry row holds the inverse pivots and, as
// columns, the rows themselves.  Two forms (RES): a part whose values and columns fit in shared
// memory beside its vectors (up to ~900 rows of a triangular mesh) loads them once, by bulk
// copies; a larger part reads them from L2 in every iteration, coalesced, a slice's loads issued
// together and (sweeps) before the barrier that its row sums wait for.
//
// What bounds it: FP64 issue and the latency between grid-wide steps.  GB300 takes 64 clocks per
// FP64 warp instruction on an SM sub-partition, with no latency beyond that, so a few warps per
// sub-partition keep the pipe busy and more only make barriers and block sums dearer
// (__syncthreads 75 clocks at 1,024 threads, 43 at 512).  Reductions use few dependent FP64
// instructions (a butterfly step is 128 clocks, a division 666, a square root 600: the tests
// compare squares).  Measured, us per iteration, the kernel with waits in the sweeps -> this one,
// cylinder pressure matrix:
//   125,364 rows: IC(0) 29.8 -> 14.1, mixed IC(0) 27.5 -> 12.1, Jacobi 15.9 -> 9.9
//   499,288 rows: IC(0) 43.5 -> 36.5, mixed IC(0) 34.1 -> 23.9, Jacobi 28.4 -> 20.6
// (FP64 issue alone: ~18 us per IC(0) iteration at 499,288 rows, ~5 at 125,364.)
#pragma once

namespace pf2 {

constexpr int kHaloWarps = 16;
constexpr int kHaloThreads = 32 * kHaloWarps;
constexpr unsigned short kHaloNone = 0xffff;   // padding row of a slice
constexpr unsigned short kHaloPubT = 0x8000;   // the row's t is published
constexpr int kHaloMaxLocal = 0x7fff;          // local rows of a part
constexpr int kHaloItem = 8;                   // entry rows per item
constexpr unsigned char kHaloLast = 0x80;      // item byte: entry rows, and whether it ends its slice

struct PartHalo {
    int P, ng;
    int R;                      // largest number of own rows
    int RL;                     // largest number of local rows (own + halo)
    int TL;                     // largest number of items of a part
    int E;                      // largest number of entry rows of a part (resident)
    const int* qs;              // own group starts (PartCg::qs)
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
    const unsigned char* pub;   // own rows: 1 where q (and r) is read by another part
    const int* ioff;            // P + 1: the parts' items in item
    const unsigned char* item;  // entry rows of an item | kHaloLast
    const int* wit;             // at (part * kHaloWarps + warp) * 2: the warp's first item (from the part's)
                                // and its first SpMV item
    const int* went;            // P * kHaloWarps + 1: the warps' first entry row in the streams
    const int* gsl;             // part k, at k (2 ng): numbers of slices of the forward and backward groups
    const unsigned short* col;  // streams: 32 entries per entry row
    const double* val;
    const int* qa;              // Q row -> row of A
    const double* diag;         // Jacobi / none: diagonal entries of the local rows, at qs[k ng] + hoff[k]
    double* x;
    const float* val32;
    unsigned long long* gq;     // packets (zeroed before the launch): published q (r at the start and
    unsigned long long* gt;     // at refinements) and t; 2 n each, alternate exchanges take alternate halves
};

template <class V> struct HaloVecs;
template <> struct HaloVecs<double> {
    __device__ static const double* val(const PartHalo& C) { return C.val; }
};
template <> struct HaloVecs<float> {
    __device__ static const float* val(const PartHalo& C) { return C.val32; }
};

// ------------------------------------------------------------ exchanges
// A value with the number of its exchange in one 16-byte (FP64) or 8-byte (FP32) word, stored and
// loaded whole: the reader sees that the value is the one it waits for, so neither a fence nor a
// counter orders an exchange (an arrival with a gpu-scope release costs ~700 clocks, the poll of
// a counter and the read behind it ~700 each).  Alternate exchanges use alternate halves, so a
// half is written again two exchanges later, when its readers have long contributed to a
// reduction that the writer has waited for, with values that depend on what they read.
template <class V> struct HaloPacket;
template <> struct HaloPacket<double> {
    static constexpr int kWords = 2;
    __device__ static __forceinline__ void put(unsigned long long* p, double v, unsigned seq) {
        asm volatile(
            "{\n\t.reg .b128 x;\n\tmov.b128 x, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], x;\n\t}"
            :
            : "l"(p), "l"(__double_as_longlong(v)), "l"((long long)seq)
            : "memory");
    }
    __device__ static __forceinline__ bool get(const unsigned long long* p, double& v, unsigned seq) {
        long long a, b;
        asm volatile(
            "{\n\t.reg .b128 x;\n\tld.relaxed.gpu.global.b128 x, [%2];\n\tmov.b128 {%0, %1}, x;\n\t}"
            : "=l"(a), "=l"(b)
            : "l"(p)
            : "memory");
        v = __longlong_as_double(a);
        return (unsigned)b == seq;
    }
};
template <> struct HaloPacket<float> {
    static constexpr int kWords = 1;
    __device__ static __forceinline__ void put(unsigned long long* p, float v, unsigned seq) {
        const unsigned long long x = (unsigned long long)seq << 32 | __float_as_uint(v);
        asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(x) : "memory");
    }
    __device__ static __forceinline__ bool get(const unsigned long long* p, float& v, unsigned seq) {
        unsigned long long x;
        asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(x) : "l"(p) : "memory");
        v = __uint_as_float((unsigned)x);
        return (unsigned)(x >> 32) == seq;
    }
};

// The packet's value once it has arrived (bounded; a wait that runs out records DEV_TIMEOUT and
// yields 0: the kernel returns at its next grid-wide step).
template <class V>
__device__ __forceinline__ V halo_settle(const unsigned long long* p, bool here, V v, unsigned seq, const GridBarrier& b,
                                         int kind, int what) {
    long long polls = 0;
    while (!here) {
        if (++polls > (b.max_polls > 0 ? b.max_polls : kFlagPolls)) {
            atomicExch(b.err, (int)DEV_TIMEOUT);
            record_timeout(b.rec, kind, kind == 1 ? (int)blockIdx.x : what, kind == 1 ? (int)seq : what, (int)seq, 0);
            return V(0);
        }
        if ((polls & 255) == 0 && *(volatile int*)b.err != 0) return V(0);
        here = HaloPacket<V>::get(p, v, seq);
    }
    return v;
}

// ------------------------------------------------------------ resident entries
__device__ __forceinline__ unsigned halo_smem_u32(const void* p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

constexpr long long kHaloCopyPolls = 1ll << 22;

// Bounded wait for phase `parity` of an mbarrier.  False where the limit ran out: it then has waited
// as long again, as the copies may still have been writing.
__device__ __forceinline__ bool halo_mbar_wait(unsigned mbar, unsigned parity) {
    for (long long i = 0; i < 2 * kHaloCopyPolls; ++i) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return i < kHaloCopyPolls;
    }
    return false;
}

__device__ __forceinline__ void halo_bulk_copy(unsigned dst, const void* src, unsigned bytes, unsigned mbar) {
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :
                 : "r"(dst), "l"(src), "r"(bytes), "r"(mbar)
                 : "memory");
}

// A warp's items in order, from this lane's values and columns of the first entry row on.
template <class V, bool RES>
struct HaloItems {
    const unsigned char *i0, *item;
    const V *v0, *v;
    const unsigned short *c0, *c;
    __device__ __forceinline__ void begin() {
        item = i0;
        v = v0;
        c = c0;
    }
    __device__ __forceinline__ V value(int k) const { return RES ? v[32 * k] : __ldg(&v[32 * k]); }
    __device__ __forceinline__ int column(int k) const { return RES ? c[32 * k] : __ldg(&c[32 * k]); }
    __device__ __forceinline__ void next() {
        const int n = (*item++ & 0x7f) * 32;
        v += n;
        c += n;
    }
};

// A part in shared memory: r, p, q, t (z shares t's array; Jacobi / none: t = 1 / a_ii and z
// apart) over the local rows, the mixed solver's update d over the own rows, the reduction
// scratch, the groups' slice counts, the own rows' publication flags, the item bytes and (RES)
// the entry rows.
template <class V, bool RES>
struct HaloSm {
    V *r, *p, *q, *t, *z, *d;
    double* red;
    const int* gsl;
    const unsigned char* pub;
    const int* hq;   // the part's halo rows
    int p0, np, nh, n, nsl;
    unsigned target; // arrivals that complete the next grid barrier
    unsigned qs, ts, rs;  // numbers of the last exchanges of q and t and of the last reduction
    // the exchanged rows of this thread's first pass (fetches without a look-up load before them)
    int nf, f_l, f_g, nz, z_l, z_g;
    HaloItems<V, RES> items;
};

constexpr int kHaloRedDoubles = 2 * kHaloThreads;
__host__ __device__ constexpr size_t halo_vec_bytes(int R, int RL, bool tri, size_t vsz, bool mixed) {
    return ((size_t)(4 + (tri ? 0 : 1)) * RL * vsz + (mixed ? (size_t)R * vsz : 0) + 127) / 128 * 128;
}
// (E: the part's entry rows when they are resident, else 0)
__host__ __device__ constexpr size_t halo_smem_bytes(int R, int RL, int TL, int ng, bool tri, size_t vsz, bool mixed,
                                                     int E) {
    return (halo_vec_bytes(R, RL, tri, vsz, mixed) + (size_t)E * 32 * (vsz + 2) + sizeof(double) * kHaloRedDoubles +
            sizeof(int) * 2 * (size_t)ng + (size_t)R + (size_t)TL + 15) / 16 * 16;
}

template <class V, bool RES>
__device__ __forceinline__ HaloSm<V, RES> halo_sm(const PartHalo& C, int n, unsigned char* base, bool tri, bool mixed,
                                                  int* err) {
    __shared__ unsigned long long mbar;
    HaloSm<V, RES> S;
    const int k = blockIdx.x, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    S.n = n;
    S.p0 = C.qs[k * C.ng];
    S.np = C.qs[(k + 1) * C.ng] - S.p0;
    S.nsl = (S.np + 31) / 32;
    const int h0 = C.hoff[k];
    S.nh = C.hoff[k + 1] - h0;
    S.hq = C.hq + h0;
    S.target = S.qs = S.ts = S.rs = 0;
    V* v = reinterpret_cast<V*>(base);
    S.r = v;
    S.p = v + C.RL;
    S.q = v + 2 * C.RL;
    S.t = v + 3 * C.RL;
    S.z = tri ? S.t : v + 4 * C.RL;
    S.d = mixed ? v + (tri ? 4 : 5) * C.RL : nullptr;
    unsigned char* entries = base + halo_vec_bytes(C.R, C.RL, tri, sizeof(V), mixed);
    S.red = reinterpret_cast<double*>(entries + (RES ? (size_t)C.E * 32 * (sizeof(V) + 2) : 0));
    int* gsl = reinterpret_cast<int*>(S.red + kHaloRedDoubles);
    unsigned char* pub = reinterpret_cast<unsigned char*>(gsl + 2 * C.ng);
    unsigned char* item = pub + C.R;
    const int i0 = C.ioff[k], ni = C.ioff[k + 1] - i0;
    for (int i = tid; i < ni; i += kHaloThreads) item[i] = C.item[i0 + i];
    for (int i = tid; i < 2 * C.ng; i += kHaloThreads) gsl[i] = C.gsl[k * 2 * C.ng + i];
    for (int l = tid; l < S.np; l += kHaloThreads) pub[l] = C.pub[S.p0 + l];
    S.gsl = gsl;
    S.pub = pub;
    S.items.i0 = item + C.wit[2 * (k * kHaloWarps + w)];
    const int ew = C.went[k * kHaloWarps + w];  // the warp's first entry row
    if constexpr (RES) {
        // all entry rows of the part, values then columns, in bulk copies of 16 KB
        const unsigned m = halo_smem_u32(&mbar);
        if (tid == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(m));
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
        const int e0 = C.went[k * kHaloWarps], e1 = C.went[(k + 1) * kHaloWarps];
        unsigned char* cols = entries + (size_t)C.E * 32 * sizeof(V);
        if (tid == 0) {
            const unsigned vb = (unsigned)(e1 - e0) * 32 * sizeof(V), cb = (unsigned)(e1 - e0) * 64;
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(m), "r"(vb + cb) : "memory");
            const unsigned char* gv = reinterpret_cast<const unsigned char*>(HaloVecs<V>::val(C) + (size_t)e0 * 32);
            const unsigned char* gc = reinterpret_cast<const unsigned char*>(C.col + (size_t)e0 * 32);
            for (unsigned o = 0; o < vb; o += 16384) halo_bulk_copy(halo_smem_u32(entries) + o, gv + o, min(16384u, vb - o), m);
            for (unsigned o = 0; o < cb; o += 16384) halo_bulk_copy(halo_smem_u32(cols) + o, gc + o, min(16384u, cb - o), m);
        }
        if (!halo_mbar_wait(m, 0)) atomicExch(err, (int)DEV_TIMEOUT);
        S.items.v0 = reinterpret_cast<const V*>(entries) + (size_t)(ew - e0) * 32 + lane;
        S.items.c0 = reinterpret_cast<const unsigned short*>(cols) + (size_t)(ew - e0) * 32 + lane;
    } else {
        S.items.v0 = HaloVecs<V>::val(C) + (size_t)ew * 32 + lane;
        S.items.c0 = C.col + (size_t)ew * 32 + lane;
    }
    S.items.begin();
    const int f0 = C.foff[k], z0 = C.zoff[k];
    S.nf = C.foff[k + 1] - f0;
    S.nz = C.zoff[k + 1] - z0;
    S.f_l = S.f_g = S.z_l = S.z_g = 0;
    const int fi = tid - 64;  // warps 0 and 1 sum the partials while the others fetch
    if (fi >= 0 && fi < S.nf) {
        S.f_l = C.fl[f0 + fi];
        S.f_g = C.fg[f0 + fi];
    }
    if (tid < S.nz) {
        S.z_l = C.zl[z0 + tid];
        S.z_g = C.zg[z0 + tid];
    }
    __syncthreads();  // the tables are in place
    return S;
}

// Row in Q order of local row l.
template <class V, bool RES>
__device__ __forceinline__ int halo_global(const HaloSm<V, RES>& S, int l) {
    return l < S.np ? S.p0 + l : __ldg(&S.hq[l - S.np]);
}

// ------------------------------------------------------------ grid-wide steps
// GridBarrier's counter with the arrivals counted here (`target` grows by the arrivals of each
// step), so no read of the counter precedes an arrival, and the error word is loaded beside the
// first poll instead of after the last.  Thread 0 waits; false on a timeout or an error.
template <bool ACQUIRE>
__device__ __forceinline__ bool halo_poll(const GridBarrier& b, unsigned target) {
    const long long limit = b.max_polls > 0 ? b.max_polls : kBarrierPolls;
    int e = *(volatile int*)b.err;
    long long polls = 0;
    unsigned c;
    while ((int)((c = ACQUIRE ? ld_acquire_gpu(b.count) : ld_relaxed_gpu(b.count)) - target) < 0) {
        if (++polls > limit) {
            atomicExch(b.err, (int)DEV_TIMEOUT);
            record_timeout(b.rec, 1, (int)blockIdx.x, (int)(target / gridDim.x) - 1, (int)c, 0);
            return false;
        }
        if ((polls & 255) == 0 && (e = *(volatile int*)b.err) != 0) return false;
    }
    return e == 0;
}

template <class V, bool RES>
__device__ __forceinline__ bool halo_sync(const GridBarrier& b, HaloSm<V, RES>& S) {
    S.target += gridDim.x;
    __syncthreads();
    int ok = 1;
    if (threadIdx.x == 0) {
        arrive_release_gpu(b.count);
        ok = halo_poll<true>(b, S.target);
    }
    return __syncthreads_and(ok);
}

// Arrival at a reduction of two values: 64 threads per value add eight threads' values each,
// then one warp per value adds two and a butterfly; its lane 0 puts the block's sum.
template <class V, bool RES>
__device__ __forceinline__ unsigned long long* halo_slot(const GridBarrier& b, const HaloSm<V, RES>& S, int value, int block) {
    return reinterpret_cast<unsigned long long*>(b.part) + 2 * (((S.rs & 1u) * 2 + value) * (size_t)gridDim.x + block);
}
template <class V, bool RES>
__device__ __forceinline__ void halo_arrive(const GridBarrier& b, HaloSm<V, RES>& S, double v0, double v1) {
    constexpr int T = kHaloThreads, Q = 64, M = T / Q;
    static_assert(T % Q == 0 && M >= 2, "block size of the tree");
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    S.red[tid] = v0;
    S.red[T + tid] = v1;
    __syncthreads();
    if (tid < 2 * Q) {
        double* c = S.red + (tid / Q) * T + tid % Q;
        double s = c[0];
#pragma unroll
        for (int i = 1; i < M; ++i) s += c[i * Q];
        c[0] = s;
    }
    __syncthreads();
    ++S.rs;
    if (w < 2) {
        const double* c = S.red + w * T + lane;
        const double s = warp_sum(c[0] + c[32]);
        if (lane == 0) {
            HaloPacket<double>::put(halo_slot(b, S, w, blockIdx.x), s, S.rs);
            asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" : : "l"(b.count) : "memory");
        }
    }
    S.target += 2 * gridDim.x;
}

// Blocks from which on a wait watches the arrival counter (one word, no ordering asked of it)
// before it reads the packets: every block polling every block's packets slows the stores it
// waits for (us per iteration without and with the counter: 152 blocks, 125,364 rows, Jacobi
// 11.0 / 10.0, IC(0) 16.4 / 14.1; 32 blocks, 16,705 rows, Jacobi 9.0 / 9.7, IC(0) 12.9 / 13.4).
constexpr unsigned kHaloCountBlocks = 64;

// The wait: warp j takes value j's sums of all blocks, adds them in block order (lane l: l, l +
// 32, ...; butterfly) and its lane 0 runs post(j, total, out) (out: the block's scalars), while
// side() runs on the warps from 2 on.  sh: totals at [16 + j], out at [24].  watch: the others'
// sums may be a while off.  False on a timeout or an error anywhere.
template <class V, bool RES, class Post, class Side>
__device__ __forceinline__ bool halo_wait(const GridBarrier& b, HaloSm<V, RES>& S, double* sh, bool watch, Post post,
                                          Side side) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    int ok = 1;
    if (w < 2) {
        if (watch && gridDim.x >= kHaloCountBlocks) {
            if (lane == 0) ok = halo_poll<false>(b, S.target);
            __syncwarp();
        }
        if (tid == 0) ok = ok && *(volatile int*)b.err == 0;
        constexpr int N = 5;
        double t = 0.0;
        for (int q0 = lane; q0 < (int)gridDim.x; q0 += 32 * N) {
            double v[N];
            bool here[N];
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const int q = q0 + 32 * i;
                here[i] = true;
                v[i] = 0.0;
                if (q < (int)gridDim.x) here[i] = HaloPacket<double>::get(halo_slot(b, S, w, q), v[i], S.rs);
            }
#pragma unroll
            for (int i = 0; i < N; ++i)
                if (q0 + 32 * i < (int)gridDim.x)
                    t += halo_settle(halo_slot(b, S, w, q0 + 32 * i), here[i], v[i], S.rs, b, 1, 0);
        }
        __syncwarp();
        t = warp_sum(t);
        if (lane == 0) {
            sh[16 + w] = t;
            post(w, t, sh + 24);
        }
        if (tid == 0) ok = ok && *(volatile int*)b.err == 0;
    } else {
        side();
    }
    return __syncthreads_and(ok);
}

template <class V, bool RES, class Post, class Side>
__device__ __forceinline__ bool halo_reduce(const GridBarrier& b, HaloSm<V, RES>& S, double v0, double v1, double* sh,
                                            Post post, Side side) {
    halo_arrive(b, S, v0, v1);
    return halo_wait(b, S, sh, true, post, side);
}

// ------------------------------------------------------------ rows
// The entry rows [lead, n) of an item in registers, and s +- sum_k f_k x[col_k] over them in
// order as a chain of fused multiply-adds.  n is uniform over the warp: the switches keep the
// loads of a slice together and the chain free of tests.
template <class V>
struct HaloEntries {
    V f[kHaloItem];
    int c[kHaloItem];
};
template <int N, class V, bool RES>
__device__ __forceinline__ void halo_load_n(const HaloItems<V, RES>& I, int lead, HaloEntries<V>& E) {
#pragma unroll
    for (int k = 0; k < N; ++k) E.f[k] = I.value(lead + k);
#pragma unroll
    for (int k = 0; k < N; ++k) E.c[k] = I.column(lead + k);
}
template <int N, bool NEG, class V>
__device__ __forceinline__ V halo_chain_n(const HaloEntries<V>& E, const V* x, V s) {
    V y[N];
#pragma unroll
    for (int k = 0; k < N; ++k) y[k] = x[E.c[k]];
#pragma unroll
    for (int k = 0; k < N; ++k) s = fma_rn(NEG ? -E.f[k] : E.f[k], y[k], s);
    return s;
}
#define PF2_HALO_CASES(X) \
    case 1: X(1); break;  \
    case 2: X(2); break;  \
    case 3: X(3); break;  \
    case 4: X(4); break;  \
    case 5: X(5); break;  \
    case 6: X(6); break;  \
    case 7: X(7); break;  \
    case 8: X(8); break;
template <class V, bool RES>
__device__ __forceinline__ void halo_load(const HaloItems<V, RES>& I, int lead, int n, HaloEntries<V>& E) {
    switch (n - lead) {
#define PF2_X(N) halo_load_n<N>(I, lead, E)
        PF2_HALO_CASES(PF2_X)
#undef PF2_X
    }
}
template <bool NEG, class V>
__device__ __forceinline__ V halo_chain(int n, const HaloEntries<V>& E, const V* x, V s) {
    switch (n) {
#define PF2_X(N) s = halo_chain_n<N, NEG>(E, x, s)
        PF2_HALO_CASES(PF2_X)
#undef PF2_X
    }
    return s;
}
// ... straight from the resident entry rows
template <int N, bool NEG, class V>
__device__ __forceinline__ V halo_chain_at_n(const V* v, const unsigned short* c, const V* x, V s) {
    V f[N], y[N];
#pragma unroll
    for (int k = 0; k < N; ++k) f[k] = v[32 * k];
#pragma unroll
    for (int k = 0; k < N; ++k) y[k] = x[c[32 * k]];
#pragma unroll
    for (int k = 0; k < N; ++k) s = fma_rn(NEG ? -f[k] : f[k], y[k], s);
    return s;
}
template <bool NEG, class V>
__device__ __forceinline__ V halo_chain_at(int n, const V* v, const unsigned short* c, const V* x, V s) {
    switch (n) {
#define PF2_X(N) s = halo_chain_at_n<N, NEG>(v, c, x, s)
        PF2_HALO_CASES(PF2_X)
#undef PF2_X
    }
    return s;
}
#undef PF2_HALO_CASES

// The packet of row j in the half of exchange seq.
template <class V, bool RES>
__device__ __forceinline__ unsigned long long* halo_row(unsigned long long* g, const HaloSm<V, RES>& S, unsigned seq, int j) {
    return g + ((size_t)(seq & 1u) * S.n + j) * HaloPacket<V>::kWords;
}

// q = A p over the part's rows (each row's entries in A's order); the rows that are F rows
// elsewhere are published.  Returns the thread's p.q terms in FP64.
template <class V, bool RES>
__device__ __forceinline__ double halo_spmv(const PartHalo& C, HaloSm<V, RES>& S) {
    unsigned long long* gq = halo_row(C.gq, S, ++S.qs, S.p0);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double pq = 0.0;
#pragma unroll 1
    for (int s = w; s < S.nsl; s += kHaloWarps) {
        const int l = s * 32 + lane;
        V acc = V(0);
        unsigned char it;
        do {
            it = *S.items.item;
            if constexpr (RES) {
                acc = halo_chain_at<false>(it & 0x7f, S.items.v, S.items.c, S.p, acc);
            } else {
                HaloEntries<V> E;
                halo_load(S.items, 0, it & 0x7f, E);
                acc = halo_chain<false>(it & 0x7f, E, S.p, acc);
            }
            S.items.next();
        } while (!(it & kHaloLast));
        if (l < S.np) {
            S.q[l] = acc;
            if (S.pub[l]) HaloPacket<V>::put(gq + (size_t)l * HaloPacket<V>::kWords, acc, S.qs);
            pq += (double)S.p[l] * (double)acc;
        }
    }
    return pq;
}

// dst of the part's F rows from the last published values, by the threads from 64 on.
template <class V, bool RES>
__device__ __forceinline__ void halo_fetch(const PartHalo& C, const HaloSm<V, RES>& S, const GridBarrier& b, V* dst) {
    const unsigned long long* gq = halo_row(C.gq, S, S.qs, 0);
    const int fi = (int)threadIdx.x - 64;
    if (fi < 0) return;
    auto take = [&](int l, int j) {
        const unsigned long long* p = gq + (size_t)j * HaloPacket<V>::kWords;
        V v;
        const bool here = HaloPacket<V>::get(p, v, S.qs);
        dst[l] = halo_settle(p, here, v, S.qs, b, 2, j);
    };
    if (fi < S.nf) take(S.f_l, S.f_g);
    for (int i = fi + kHaloThreads - 64, f0 = __ldg(&C.foff[blockIdx.x]); i < S.nf; i += kHaloThreads - 64)
        take(__ldg(&C.fl[f0 + i]), __ldg(&C.fg[f0 + i]));
}

// A slice of a sweep: head(row) gives the chain's start for the lane's row (kHaloNone: padding;
// it may wait for a barrier), tail(row, sum, pivot) takes s - sum_k f_k x[col_k] over the row's
// entries in entry order.
template <class V, bool RES, class Head, class Tail>
__device__ __forceinline__ void halo_slice(HaloItems<V, RES>& I, const V* x, Head head, Tail tail) {
    unsigned char it = *I.item;
    const V piv = I.value(0);
    const int row = I.column(0);
    V s;
    if constexpr (RES) {
        s = head(row);
        s = halo_chain_at<true>((it & 0x7f) - 1, I.v + 32, I.c + 32, x, s);
        while (!(it & kHaloLast)) {
            I.next();
            it = *I.item;
            s = halo_chain_at<true>(it & 0x7f, I.v, I.c, x, s);
        }
        tail(row, s, piv);
        I.next();
        return;
    }
    HaloEntries<V> E;
    halo_load(I, 1, it & 0x7f, E);
    I.next();
    s = head(row);
    s = halo_chain<true>((it & 0x7f) - 1, E, x, s);
    while (!(it & kHaloLast)) {
        it = *I.item;
        halo_load(I, 0, it & 0x7f, E);
        I.next();
        s = halo_chain<true>(it & 0x7f, E, x, s);
    }
    tail(row, s, piv);
}

// Forward sweep over the own rows and the F rows, group by group: r -= alpha q, t = L^{-1} r
// (alpha = 0 with q = 0 leaves r as it is).  Own t that is read elsewhere is published.
// Returns the own rows' r.r (want_rr) and (IC) t.t terms.
template <bool IC, class V, bool RES>
__device__ __forceinline__ double2 halo_fwd(const PartHalo& C, HaloSm<V, RES>& S, V alpha, bool want_rr) {
    unsigned long long* gt = halo_row(C.gt, S, ++S.ts, S.p0);
    const int w = threadIdx.x >> 5;
    double rr = 0.0, tt = 0.0;
    S.items.begin();
#pragma unroll 1
    for (int g = 0; g < C.ng; ++g) {
        const int ns = S.gsl[g];
        bool wait = g > 0;  // for the part's earlier groups, once
#pragma unroll 1
        for (int s = w; s < ns; s += kHaloWarps) {
            V ra = V(0);
            halo_slice(S.items, S.t, [&](int row) {
                if (row != kHaloNone) {  // the update of r needs no earlier group: before the barrier
                    const int l = row & kHaloMaxLocal;
                    ra = fma_rn(-alpha, S.q[l], S.r[l]);
                    S.r[l] = ra;
                }
                __syncwarp();
                if (wait) __syncthreads();
                wait = false;
                return ra;
            }, [&](int row, V rest, V piv) {
                if (row == kHaloNone) return;
                const int l = row & kHaloMaxLocal;
                const V v = IC ? rest * piv : rest;
                S.t[l] = v;
                if (row & kHaloPubT) HaloPacket<V>::put(gt + (size_t)l * HaloPacket<V>::kWords, v, S.ts);
                if (l < S.np) {
                    if (want_rr) rr += (double)ra * (double)ra;
                    if (IC) tt += (double)v * (double)v;
                }
            });
        }
        if (wait) __syncthreads();
    }
    return make_double2(rr, tt);
}

// t of the Z rows that are not F rows, from their owners.  work() runs between the first load
// and its use.
template <class V, bool RES, class Work>
__device__ __forceinline__ void halo_fetch_t(const PartHalo& C, HaloSm<V, RES>& S, const GridBarrier& b, Work work) {
    const unsigned long long* gt = halo_row(C.gt, S, S.ts, 0);
    const bool mine = (int)threadIdx.x < S.nz;
    const unsigned long long* p0 = gt + (size_t)S.z_g * HaloPacket<V>::kWords;
    V v0 = V(0);
    bool here = false;
    if (mine) here = HaloPacket<V>::get(p0, v0, S.ts);
    work();
    if (mine) S.t[S.z_l] = halo_settle(p0, here, v0, S.ts, b, 2, S.z_g);
    for (int i = threadIdx.x + kHaloThreads, z0 = __ldg(&C.zoff[blockIdx.x]); i < S.nz; i += kHaloThreads) {
        const int j = __ldg(&C.zg[z0 + i]);
        const unsigned long long* p = gt + (size_t)j * HaloPacket<V>::kWords;
        V v;
        const bool h = HaloPacket<V>::get(p, v, S.ts);
        S.t[__ldg(&C.zl[z0 + i])] = halo_settle(p, h, v, S.ts, b, 2, j);
    }
}

// Backward sweep over the own rows and the Z rows: z = U^{-1} t in t's array.  Returns the own
// rows' r.z terms (want_rz).
template <class V, bool RES>
__device__ __forceinline__ double halo_bwd(const PartHalo& C, HaloSm<V, RES>& S, bool want_rz) {
    const int w = threadIdx.x >> 5;
    double rz = 0.0;
#pragma unroll 1
    for (int g = C.ng - 1; g >= 0; --g) {
        const int ns = S.gsl[C.ng + g];
        bool wait = true;  // for the part's later groups and the fetched t, once
#pragma unroll 1
        for (int s = w; s < ns; s += kHaloWarps) {
            halo_slice(S.items, S.z, [&](int row) {
                __syncwarp();
                if (wait) __syncthreads();
                wait = false;
                return row != kHaloNone ? S.t[row] : V(0);
            }, [&](int row, V rest, V piv) {
                if (row == kHaloNone) return;
                const V v = rest * piv;
                S.z[row] = v;
                if (want_rz && row < S.np) rz += (double)S.r[row] * (double)v;
            });
        }
        if (wait) __syncthreads();
    }
    return rz;
}

// p = z + beta p on the own rows and ring 1.  No barrier inside; the SpMV that follows needs one.
template <class V, bool RES>
__device__ __forceinline__ void halo_p_update(const PartHalo& C, const HaloSm<V, RES>& S, V beta) {
    const int k = blockIdx.x;
    const int a0 = __ldg(&C.r1off[k]), nr = __ldg(&C.r1off[k + 1]) - a0;
    for (int i = threadIdx.x; i < S.np + nr; i += kHaloThreads) {
        const int l = i < S.np ? i : (int)__ldg(&C.r1[a0 + i - S.np]);
        S.p[l] = fma_rn(beta, S.p[l], S.z[l]);
    }
}

// r = b - A x in FP64 over the part's rows (x from the global iterate in Q order), published for
// the parts that hold it as halo: store(l, r).  Returns the b.b and r.r terms.
template <class V, bool RES, class Store>
__device__ __forceinline__ double2 halo_residual(const KArgs& a, const PartHalo& C, const HaloSm<V, RES>& S, Store store) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, wk = blockIdx.x * kHaloWarps + w;
    const int i0 = C.wit[2 * wk], i1 = C.wit[2 * wk + 1];
    int row = C.went[wk], i = i1 - i0;
    const unsigned char* item = S.items.i0;
    for (int j = 0; j < i; ++j) row += item[j] & 0x7f;
    double bb = 0.0, rr = 0.0;
    for (int s = w; s < S.nsl; s += kHaloWarps) {
        const int l = s * 32 + lane;
        double v = 0.0;
        unsigned char it;
        do {
            it = item[i++];
            for (int k = 0; k < (it & 0x7f); ++k, ++row) {
                const size_t e = (size_t)row * 32 + lane;
                if (l < S.np) v = __fma_rn(__ldg(&C.val[e]), __ldcg(&C.x[halo_global(S, (int)__ldg(&C.col[e]))]), v);
            }
        } while (!(it & kHaloLast));
        if (l < S.np) {
            const double bi = a.b[__ldg(&C.qa[S.p0 + l])];
            const double ri = bi - v;
            store(l, ri);
            bb += bi * bi;
            rr += ri * ri;
        }
    }
    return make_double2(bb, rr);
}

struct HaloNoSide {
    __device__ void operator()() const {}
};
struct HaloNoPost {
    __device__ void operator()(int, double, double*) const {}
};

// FP64 CG: MODE 0 Jacobi or no preconditioner, 1 IC(0), 2 ILU(0) (pcg_part's iterations).  The
// loop starts at the preconditioner with alpha = beta = 0 and p = q = 0, which leaves r and x
// as they are and makes p = z.
template <int MODE, bool RES>
__device__ __forceinline__ void pcg_halo(const KArgs& a, const PartHalo& C, HaloSm<double, RES>& S, double* sh) {
    const int tid = threadIdx.x, np = S.np;
    constexpr int T = kHaloThreads;
    const bool rel = a.criterion == PF2_CRITERION_REL;
    const bool jac = a.precond == PF2_PRECOND_JACOBI;
    for (int l = tid; l < np; l += T) __stcg(&C.x[S.p0 + l], a.x[__ldg(&C.qa[S.p0 + l])]);
    for (int l = tid; l < np + S.nh; l += T) {
        S.p[l] = 0.0;
        S.q[l] = 0.0;
        // (tri: finite values where a padding entry of the first sweep looks)
        S.t[l] = MODE == 0 ? 1.0 / __ldg(&C.diag[S.p0 + C.hoff[blockIdx.x] + l]) : 0.0;
    }
    if (!halo_sync(a.bar, S)) return;
    unsigned long long* gr = halo_row(C.gq, S, ++S.qs, S.p0);
    const double2 br = halo_residual(a, C, S, [&](int l, double ri) {
        S.r[l] = ri;
        if (S.pub[l]) HaloPacket<double>::put(gr + 2 * (size_t)l, ri, S.qs);
    });
    // b.b and r.r beside the fetch of the F rows' r
    if (!halo_reduce(a.bar, S, br.x, br.y, sh, HaloNoPost(), [&]() { halo_fetch(C, S, a.bar, S.r); })) return;
    const double bb_all = sh[16];
    double rr = sh[17], gamma = 1.0, alpha = 0.0;
    // the tests compare r.r or r.z with the square of the tolerance
    const double bound = rel ? (a.tol * a.tol) * bb_all : a.tol * a.tol;
    const double rr0 = rr;
    int it = 0;
    bool conv = false, first = true;
    auto post = [&](int j, double tot, double* out) {
        if (j == 0) out[1] = first ? 0.0 : tot / gamma;
        if (rel ? j == 1 : j == 0) out[0] = rel ? tot <= bound : tot < bound;
    };
    while (true) {
        // the update of x with the last alpha, beside the exchange or a reduction's wait
        auto x_update = [&]() {
            for (int l = tid; l < np; l += T)
                __stcg(&C.x[S.p0 + l], __fma_rn(alpha, S.p[l], __ldcg(&C.x[S.p0 + l])));
        };
        double rz = 0.0, r2 = 0.0;
        if (MODE == 0) {
            for (int l = tid; l < np + S.nh; l += T) {
                const double ri = __fma_rn(-alpha, S.q[l], S.r[l]);
                const double zi = jac ? ri * S.t[l] : ri;
                S.r[l] = ri;
                S.z[l] = zi;
                if (l < np) {
                    rz += ri * zi;
                    if (rel) r2 += ri * ri;
                }
            }
            halo_arrive(a.bar, S, rz, r2);
            x_update();
        } else {
            const double2 f = halo_fwd<MODE == 1>(C, S, alpha, rel);
            // IC(0): z = L^{-T} t does not depend on beta, so the x update and the backward sweep run
            // between the arrival at the t.t (and r.r) reduction and the wait for the others
            if (MODE == 1) halo_arrive(a.bar, S, f.y, f.x);
            halo_fetch_t(C, S, a.bar, x_update);
            rz = halo_bwd(C, S, MODE == 2);
            if (MODE == 2) halo_arrive(a.bar, S, rz, f.x);
        }
        if (!halo_wait(a.bar, S, sh, MODE != 1, post, HaloNoSide())) return;
        gamma = sh[16];
        if (rel) rr = sh[17];
        first = false;
        if (sh[24] != 0.0) { conv = true; break; }
        if (it >= a.maxit) break;
        ++it;
        halo_p_update(C, S, sh[25]);
        __syncthreads();
        if (MODE == 0) S.items.begin();
        const double pq = halo_spmv(C, S);
        // alpha beside the fetch of the F rows' q
        if (!halo_reduce(a.bar, S, pq, 0.0, sh,
                         [&](int j, double tot, double* out) { if (j == 0) out[0] = gamma / tot; },
                         [&]() { halo_fetch(C, S, a.bar, S.q); }))
            return;
        alpha = sh[24];
    }
    if (!rel && it > 0) {  // with the absolute criterion (a test of r.z alone) r.r is reduced once, here
        double f = 0.0;
        for (int l = tid; l < np; l += T) f += S.r[l] * S.r[l];
        if (!halo_reduce(a.bar, S, f, 0.0, sh, HaloNoPost(), HaloNoSide())) return;
        rr = sh[16];
    }
    if (it == 0) rr = rr0;
    for (int l = tid; l < np; l += T) a.x[__ldg(&C.qa[S.p0 + l])] = __ldcg(&C.x[S.p0 + l]);
    if (blockIdx.x == 0 && tid == 0) {
        const double bnorm = sqrt(bb_all);
        a.out->iterations = it;
        a.out->converged = conv ? 1 : 0;
        a.out->residual = rel ? sqrt(rr) / (bnorm > 0 ? bnorm : 1.0) : sqrt(gamma);
        a.out->relres = sqrt(rr) / (bnorm > 0 ? bnorm : 1.0);
        a.out->status = conv ? DEV_OK : DEV_NOT_CONVERGED;
    }
}

// Mixed-precision CG (pcg_part_mixed's algorithm: FP32 iteration, FP64 sums, reliable updates).
// Passes of the loop: the first (preconditioner of r, gamma = r.z), ordinary ones, and after a
// refinement one more preconditioner with the true residual, which gives the next beta.
template <bool IC, bool RES>
__device__ __forceinline__ void pcg_halo_mixed(const KArgs& a, const PartHalo& C, HaloSm<float, RES>& S, double* sh) {
    const int tid = threadIdx.x, np = S.np;
    constexpr int T = kHaloThreads;
    for (int l = tid; l < np; l += T) {
        __stcg(&C.x[S.p0 + l], a.x[__ldg(&C.qa[S.p0 + l])]);
        S.d[l] = 0.0f;
    }
    for (int l = tid; l < np + S.nh; l += T) {
        S.p[l] = 0.0f;
        S.q[l] = 0.0f;
        S.t[l] = 0.0f;  // finite where a padding entry of the first sweep looks
    }
    if (!halo_sync(a.bar, S)) return;
    enum { FIRST, ORDINARY, REFINED };
    int pass = FIRST, it = 0, refinements = 0;
    double bnorm = 0.0, target = 0.0, rnorm = 0.0, rlast = 0.0, gamma = 0.0;
    float alpha = 0.0f;
    bool conv = false;
    while (true) {
        if (pass != ORDINARY) {
            // r = b - A x and the test in FP64
            unsigned long long* gr = halo_row(C.gq, S, ++S.qs, S.p0);
            const double2 br = halo_residual(a, C, S, [&](int l, double ri) {
                S.r[l] = (float)ri;
                if (S.pub[l]) HaloPacket<float>::put(gr + l, (float)ri, S.qs);
            });
            if (!halo_reduce(a.bar, S, br.x, br.y, sh, [&](int j, double tot, double* out) { out[j] = sqrt(tot); },
                             [&]() { halo_fetch(C, S, a.bar, S.r); }))
                return;
            ++refinements;
            bnorm = sh[24];
            rnorm = sh[25];
            target = a.tol * bnorm;
            rlast = rnorm;
            if (rnorm <= target) { conv = true; break; }
            alpha = 0.0f;  // the sweep takes r as it is
            if (pass == FIRST && it >= a.maxit) break;
        }
        // refinement test (squares: rit <= max(eta rlast, target)) and beta (0 in the first pass)
        const double lim = fmax(a.inner_eta * rlast, target), lim2 = lim * lim;
        auto post = [&](int j, double tot, double* out) {
            if (j == 0) out[1] = pass == FIRST ? 0.0 : (double)(float)(tot / gamma);
            else out[0] = tot <= lim2;
        };
        auto d_update = [&]() {
            if (pass == ORDINARY)
                for (int l = tid; l < np; l += T) S.d[l] = S.d[l] + alpha * S.p[l];
        };
        const double2 f = halo_fwd<IC>(C, S, alpha, pass == ORDINARY);
        // IC(0): the backward sweep (z alone) overlaps the reduction, as in pcg_halo; the first pass
        // takes gamma = r.z from the backward sweep
        const bool tt = IC && pass != FIRST;
        if (tt) halo_arrive(a.bar, S, f.y, f.x);
        halo_fetch_t(C, S, a.bar, d_update);
        const double rz = halo_bwd(C, S, !tt);
        if (!tt) halo_arrive(a.bar, S, rz, f.x);
        if (!halo_wait(a.bar, S, sh, !tt, post, HaloNoSide())) return;
        if (pass == ORDINARY && sh[24] != 0.0) {
            // refinement: x += d; the next pass recomputes r and runs the sweeps on it (the search
            // direction is kept)
            for (int l = tid; l < np; l += T) {
                __stcg(&C.x[S.p0 + l], __ldcg(&C.x[S.p0 + l]) + (double)S.d[l]);
                S.d[l] = 0.0f;
            }
            if (!halo_sync(a.bar, S)) return;
            pass = REFINED;
            continue;
        }
        gamma = sh[16];
        const float beta = (float)sh[25];
        if (pass != FIRST && it >= a.maxit) break;
        pass = ORDINARY;
        ++it;
        halo_p_update(C, S, beta);
        __syncthreads();
        const double pq = halo_spmv(C, S);
        if (!halo_reduce(a.bar, S, pq, 0.0, sh,
                         [&](int j, double tot, double* out) { if (j == 0) out[0] = (double)(float)(gamma / tot); },
                         [&]() { halo_fetch(C, S, a.bar, S.q); }))
            return;
        alpha = (float)sh[24];
    }
    if (!conv)  // iteration limit: keep the accumulated update
        for (int l = tid; l < np; l += T)
            __stcg(&C.x[S.p0 + l], __ldcg(&C.x[S.p0 + l]) + (double)S.d[l]);
    for (int l = tid; l < np; l += T) a.x[__ldg(&C.qa[S.p0 + l])] = __ldcg(&C.x[S.p0 + l]);
    if (blockIdx.x == 0 && tid == 0) {
        a.out->iterations = it;
        a.out->converged = conv ? 1 : 0;
        a.out->residual = rnorm / (bnorm > 0 ? bnorm : 1.0);
        a.out->relres = rnorm / (bnorm > 0 ? bnorm : 1.0);
        a.out->status = conv ? DEV_OK : DEV_NOT_CONVERGED;
        a.out->pad = refinements;
    }
}

template <int MODE, bool RES>
__global__ void __launch_bounds__(kHaloThreads, 1) k_pcg_halo(KArgs a, PartHalo C) {
    __shared__ double sh[kShDoubles];
    extern __shared__ __align__(128) unsigned char halo_smem[];
    HaloSm<double, RES> S = halo_sm<double, RES>(C, a.A.n, halo_smem, MODE != 0, false, a.bar.err);
    pcg_halo<MODE>(a, C, S, sh);
}

template <bool IC, bool RES>
__global__ void __launch_bounds__(kHaloThreads, 1) k_pcg_halo_mixed(KArgs a, PartHalo C) {
    __shared__ double sh[kShDoubles];
    extern __shared__ __align__(128) unsigned char halo_smem[];
    HaloSm<float, RES> S = halo_sm<float, RES>(C, a.A.n, halo_smem, true, true, a.bar.err);
    pcg_halo_mixed<IC>(a, C, S, sh);
}

}  // namespace pf2

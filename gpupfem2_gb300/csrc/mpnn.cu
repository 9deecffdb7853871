// mpnn.cu - the learned initial guess of the pressure solve (no reference counterpart).
//
// A message-passing network over the mesh graph (nodes; edges = off-diagonal CSR
// entries, symmetric) with 5 input features, 64 hidden units and 3 layers:
//   h0 = relu(W0 f + c0)
//   l = 1..3:  m_i = mean_{j in N(i)} h_j ;  h = h + relu(W_l [h ; m] + c_l)
//   y  = w4 . h + c4
// Master parameters are FP32; the per-node MLPs run on the tensor cores with BF16
// weights and activations and FP32 accumulation on tcgen05 (accumulators in tensor
// memory, 128 nodes per CTA); the mma.sync m16n8k16 kernels stay as the
// PF2_MPNN_MMA=sync path.  Training
// (backward and AdamW) runs on the device; gradients are summed in a fixed order.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "device.cuh"
#include "internal.cuh"

namespace pf2 {

constexpr int MH = 64;      // hidden width
constexpr int MIN = 5;      // input features
constexpr int ML = 3;       // message-passing layers
constexpr int MK = 2 * MH;  // layer input width [h ; m]
constexpr int kTile = 64;   // nodes per CTA tile
constexpr int kMpnnThreads = 128;
constexpr int kPad = 8;     // bf16 row padding against bank conflicts

constexpr int kParamW0 = 0;
constexpr int kParamC0 = kParamW0 + MH * MIN;
constexpr int kParamLayer0 = kParamC0 + MH;
constexpr int kLayerSize = MH * MK + MH;
constexpr int kParamW4 = kParamLayer0 + ML * kLayerSize;
constexpr int kParamC4 = kParamW4 + MH;
constexpr int kParams = kParamC4 + 1;

__device__ __forceinline__ unsigned pack_bf16(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<unsigned*>(&v);
}

// D = A(16x16, row) * B(16x8, col) + D, bf16 inputs, f32 accumulate
__device__ __forceinline__ void mma16816(float d[4], const unsigned a[4], const unsigned b[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// One warp: acc[16 x 8NT] += A[16 x 16KT] (smem row-major, stride sa) * B, with B given as
// rows of n (smem [n][k], stride sb).
template <int KT, int NT>
__device__ __forceinline__ void warp_gemm(const __nv_bfloat16* A, int sa, const __nv_bfloat16* B, int sb,
                                          float acc[NT][4]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int kt = 0; kt < KT; ++kt) {
        const int k0 = kt * 16 + 2 * t;
        unsigned a[4];
        a[0] = *reinterpret_cast<const unsigned*>(A + g * sa + k0);
        a[1] = *reinterpret_cast<const unsigned*>(A + (g + 8) * sa + k0);
        a[2] = *reinterpret_cast<const unsigned*>(A + g * sa + k0 + 8);
        a[3] = *reinterpret_cast<const unsigned*>(A + (g + 8) * sa + k0 + 8);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const __nv_bfloat16* Bn = B + (nt * 8 + g) * sb + k0;
            unsigned b[2];
            b[0] = *reinterpret_cast<const unsigned*>(Bn);
            b[1] = *reinterpret_cast<const unsigned*>(Bn + 8);
            mma16816(acc[nt], a, b);
        }
    }
}

struct Graph {
    int n;
    const int* rowptr;
    const int* col;
    const float* deg_inv;  // 1 / #neighbours (0 for an isolated node)
};

// ---------------------------------------------------------------- forward
// Node-row kernels take 16 threads per node, four features each: a row is one 256-byte access
// (a thread per node touches 32 rows with every load).
constexpr int kRowThreads = 256;
constexpr int kRowNodes = kRowThreads / 16;

// Bound by the 128 MB it writes at 499,288 nodes: 172 us with a thread per node -> 40 us.
__global__ void __launch_bounds__(kRowThreads) k_mpnn_encoder(Graph G, const float* __restrict__ feat,
                                                              const float* __restrict__ P, float* H0,
                                                              unsigned long long* mask0) {
    const int o = (threadIdx.x & 15) * 4;
    float w[4][MIN], c[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        c[j] = P[kParamC0 + o + j];
#pragma unroll
        for (int k = 0; k < MIN; ++k) w[j][k] = P[kParamW0 + (o + j) * MIN + k];
    }
    for (int base = blockIdx.x * kRowNodes; base < G.n; base += gridDim.x * kRowNodes) {
        const int i = base + (threadIdx.x >> 4);
        const bool in = i < G.n;
        float f[MIN];
#pragma unroll
        for (int k = 0; k < MIN; ++k) f[k] = in ? feat[(size_t)i * MIN + k] : 0.0f;
        float h[4];
        unsigned bits = 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float s = c[j];
#pragma unroll
            for (int k = 0; k < MIN; ++k) s += w[j][k] * f[k];
            if (s > 0.0f) bits |= 1u << ((o + j) & 31);
            h[j] = s > 0.0f ? s : 0.0f;
        }
        if (in) *reinterpret_cast<float4*>(&H0[(size_t)i * MH + o]) = make_float4(h[0], h[1], h[2], h[3]);
        // eight lanes hold a word of the node's mask
#pragma unroll
        for (int d = 1; d < 8; d <<= 1) bits |= __shfl_xor_sync(0xffffffffu, bits, d);
        if (in && (threadIdx.x & 7) == 0) reinterpret_cast<unsigned*>(mask0)[2 * (size_t)i + (o >> 5)] = bits;
    }
}

// mean of the neighbours' h (fixed order: ascending column)
__device__ __forceinline__ void gather_mean(const Graph& G, const float* __restrict__ H, int i, int o, float& out) {
    float s = 0.0f;
    for (int k = G.rowptr[i]; k < G.rowptr[i + 1]; ++k) {
        const int j = G.col[k];
        if (j != i) s += H[(size_t)j * MH + o];
    }
    out = s * G.deg_inv[i];
}

// The sum of the neighbours' rows of X at features o .. o + 3 added to s, in ascending column
// order (gather_mean's order), four columns' loads in flight together (eight cost registers that
// four CTAs per SM do not have: a pass over 499,288 nodes 2.82 ms against 2.43).
__device__ __forceinline__ float4 gather_rows(const Graph& G, const float* __restrict__ X, int i, int o, float4 s) {
    const int k1 = __ldg(&G.rowptr[i + 1]);
    for (int k = __ldg(&G.rowptr[i]); k < k1; k += 4) {
        int j[4];
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) j[u] = k + u < k1 ? __ldg(&G.col[k + u]) : i;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (j[u] != i) v[u] = __ldg(reinterpret_cast<const float4*>(&X[(size_t)j[u] * MH + o]));
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (j[u] != i) {
                s.x += v[u].x;
                s.y += v[u].y;
                s.z += v[u].z;
                s.w += v[u].w;
            }
    }
    return s;
}

// One layer: h_out = h_in + relu(W [h_in ; m] + c); stores m (for the backward pass)
// and the relu mask.  CTA = 4 warps x 16 nodes.
__global__ void __launch_bounds__(kMpnnThreads) k_mpnn_layer(Graph G, const float* __restrict__ Hin,
                                                             const __nv_bfloat16* __restrict__ Wb,
                                                             const float* __restrict__ c, float* Hout, float* M,
                                                             unsigned long long* mask) {
    __shared__ __align__(16) __nv_bfloat16 sA[kTile][MK + kPad];
    __shared__ __align__(16) __nv_bfloat16 sW[MH][MK + kPad];
    const int base = blockIdx.x * kTile;
    for (int q = threadIdx.x; q < MH * MK; q += blockDim.x) sW[q / MK][q % MK] = Wb[q];
    for (int q = threadIdx.x; q < kTile * MH; q += blockDim.x) {
        const int r = q / MH, o = q % MH, i = base + r;
        float h = 0.0f, m = 0.0f;
        if (i < G.n) {
            h = Hin[(size_t)i * MH + o];
            gather_mean(G, Hin, i, o, m);
            M[(size_t)i * MH + o] = m;
        }
        sA[r][o] = __float2bfloat16_rn(h);
        sA[r][MH + o] = __float2bfloat16_rn(m);
    }
    __syncthreads();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    float acc[MH / 8][4];
#pragma unroll
    for (int nt = 0; nt < MH / 8; ++nt)
        for (int k = 0; k < 4; ++k) acc[nt][k] = 0.0f;
    warp_gemm<MK / 16, MH / 8>(&sA[w * 16][0], MK + kPad, &sW[0][0], MK + kPad, acc);
    // epilogue: rows g, g+8 of this warp's 16 nodes; columns nt*8 + 2t, +1
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int i = base + w * 16 + g + 8 * half;
        const bool valid = i < G.n;
        unsigned long long bits = 0ull;
#pragma unroll
        for (int nt = 0; nt < MH / 8; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int o = nt * 8 + 2 * t + e;
                const float z = acc[nt][2 * half + e] + c[o];
                if (z > 0.0f) bits |= 1ull << o;
                if (valid) Hout[(size_t)i * MH + o] = Hin[(size_t)i * MH + o] + (z > 0.0f ? z : 0.0f);
            }
        // the four threads of a quad own disjoint columns of the row: combine their bits
        // (every lane takes part in the shuffles; only the store is guarded)
        bits |= __shfl_xor_sync(0xffffffffu, bits, 1);
        bits |= __shfl_xor_sync(0xffffffffu, bits, 2);
        if (valid && t == 0) mask[i] = bits;
    }
}

// ------------------------------------------------ fifth-generation tensor cores
// The layer GEMM on tcgen05: one thread issues tcgen05.mma (kind::f16, BF16 operands from
// shared memory, FP32 accumulator in tensor memory), the CTA reads the accumulator back
// with tcgen05.ld.  Operands sit in shared memory in the canonical K-major layout without
// swizzle: 8-row x 16-byte core matrices, element (r, k) of an R-row tile at byte
//   ((k / 8) * (R / 8) + r / 8) * 128 + (r % 8) * 16 + (k % 8) * 2,
// so core matrices adjacent in K are R * 16 bytes apart (the descriptor's leading byte
// offset) and those adjacent in rows 128 bytes apart (its stride byte offset).
constexpr int kTcTile = 128;  // nodes per CTA: the MMA's M (accumulator lanes 0..127)
constexpr long long kTcPolls = 1ll << 24;
// The layer kernels keep 48-53 KB of shared memory (operands, and the FP32 results staged in the
// first operand's place for coalesced rows), so four CTAs of eight warps share an SM and one
// CTA's gather or epilogue runs under another's.  CTAs are persistent: weights, tensor memory
// and the mbarrier are set up once.
constexpr int kTcThreads = 256;
constexpr int kTcCtasPerSm = 4;
constexpr int kZStride = MH + 4;                       // staged row of 64 floats (no bank conflicts by rows)
constexpr int kTcRegionZ = 35 * 1024;                  // kTcTile rows of kZStride floats, or A (32 KB)
static_assert(kTcRegionZ >= kTcTile * kZStride * 4 && kTcRegionZ >= kTcTile * MK * 2 && kTcRegionZ % 1024 == 0, "region");
constexpr int kTcSmem = kTcRegionZ + MH * MK * 2;      // + W
constexpr int kTcBwSmem = (MK + MH) * kTcTile * 2;     // [h ; m]^T and dz^T

__device__ __forceinline__ unsigned smem_u32(const void* p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ int tc_offset(int r, int k, int rows) {
    return ((k >> 3) * (rows >> 3) + (r >> 3)) * 128 + (r & 7) * 16 + (k & 7) * 2;
}

// Shared-memory matrix descriptor (no swizzle, version 1): start, leading byte offset
// (between core matrices adjacent in K), stride byte offset (adjacent in rows).
__device__ __forceinline__ unsigned long long tc_desc(unsigned addr, unsigned lbo, unsigned sbo) {
    return (unsigned long long)((addr >> 4) & 0x3FFFu) | ((unsigned long long)((lbo >> 4) & 0x3FFFu) << 16) |
           ((unsigned long long)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major,
// N and M as given.
__host__ __device__ constexpr unsigned tc_idesc(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) | ((unsigned)(m >> 4) << 24);
}

__device__ __forceinline__ void tc_mma(unsigned tmem_d, unsigned long long a, unsigned long long b, unsigned idesc,
                                       int accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        :
        : "r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void tc_commit(unsigned mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" : : "r"(mbar)
                 : "memory");
}

// Bounded wait for phase `parity` of an mbarrier; false when the limit ran out.
__device__ __forceinline__ bool mbar_wait(unsigned mbar, unsigned parity) {
    for (long long i = 0; i < kTcPolls; ++i) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// 32 consecutive accumulator columns of this warp's 32 lanes: register j of lane l holds
// row (lane base + l), column (col + j).
__device__ __forceinline__ void tc_ld32(unsigned taddr, float (&v)[32]) {
    unsigned r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,"
        "%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
}

// The CTA's tensor-memory columns (warp 0 allocates; power of two >= 32).
__device__ __forceinline__ void tc_alloc(unsigned* slot, int cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}

__device__ __forceinline__ void tc_dealloc(unsigned tmem, int cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols));
}

__device__ __forceinline__ void tc_sync_in() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// One layer as k_mpnn_layer, tiles of 128 nodes on tcgen05: h_out = h_in + relu(W [h ; m] + c), m
// (for the backward pass) and the relu mask stored.  Warp 0 holds the 64 accumulator columns of
// tensor memory; thread 0 issues the eight K = 16 MMAs (M = 128, N = 64); warp w reads back rows
// 32 (w mod 4) .. + 31, columns 32 (w / 4) .. + 31.  A wait that runs out sets *err and ends the
// CTA.  Bound by L2 and DRAM traffic (three rows of 256 B written or read per node besides the
// gathered ones).  Measured at 499,288 nodes: 1,522 us with 128 threads, one (node, feature) pair
// per thread step and two CTAs per SM (latency of the gather) -> 157 us.
__global__ void __launch_bounds__(kTcThreads, kTcCtasPerSm) k_mpnn_layer_tc(Graph G, const float* __restrict__ Hin,
                                                                            const __nv_bfloat16* __restrict__ Wb,
                                                                            const float* __restrict__ c, float* Hout,
                                                                            float* M, unsigned* mask, int* err) {
    extern __shared__ __align__(1024) unsigned char tc_smem[];
    unsigned char* sA = tc_smem;                       // [node][in], canonical layout
    float* sZ = reinterpret_cast<float*>(tc_smem);     // relu results, once the MMAs have read A
    unsigned char* sB = tc_smem + kTcRegionZ;          // W [out][in], canonical layout
    __shared__ __align__(8) unsigned long long mbar;
    __shared__ unsigned tmem_slot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) tc_alloc(&tmem_slot, MH);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar)));
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    for (int q = tid; q < MH * MK / 8; q += kTcThreads) {
        const int o = q / (MK / 8), k = q % (MK / 8) * 8;
        *reinterpret_cast<uint4*>(sB + tc_offset(o, k, MH)) = __ldg(reinterpret_cast<const uint4*>(Wb + o * MK + k));
    }
    const int ntiles = (G.n + kTcTile - 1) / kTcTile;
    unsigned phase = 0;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int base = tile * kTcTile;
        for (int q = tid; q < kTcTile * 16; q += kTcThreads) {
            const int r = q >> 4, o = (q & 15) * 4, i = base + r;
            float4 h = make_float4(0.0f, 0.0f, 0.0f, 0.0f), m = h;
            if (i < G.n) {
                h = __ldg(reinterpret_cast<const float4*>(&Hin[(size_t)i * MH + o]));
                m = gather_rows(G, Hin, i, o, m);
                const float d = __ldg(&G.deg_inv[i]);
                m = make_float4(m.x * d, m.y * d, m.z * d, m.w * d);
                *reinterpret_cast<float4*>(&M[(size_t)i * MH + o]) = m;
            }
            *reinterpret_cast<uint2*>(sA + tc_offset(r, o, kTcTile)) = make_uint2(pack_bf16(h.x, h.y), pack_bf16(h.z, h.w));
            *reinterpret_cast<uint2*>(sA + tc_offset(r, MH + o, kTcTile)) =
                make_uint2(pack_bf16(m.x, m.y), pack_bf16(m.z, m.w));
        }
        tc_sync_in();  // the operands written by threads become visible to the tensor cores' async proxy
        const unsigned tmem = tmem_slot;
        if (tid == 0) {
            const unsigned a0 = smem_u32(sA), b0 = smem_u32(sB);
            constexpr unsigned idesc = tc_idesc(kTcTile, MH);
#pragma unroll
            for (int ks = 0; ks < MK / 16; ++ks)
                tc_mma(tmem, tc_desc(a0 + ks * 2 * (kTcTile * 16), kTcTile * 16, 128),
                       tc_desc(b0 + ks * 2 * (MH * 16), MH * 16, 128), idesc, ks > 0);
            tc_commit(smem_u32(&mbar));
        }
        // every thread polls; the outcome is made block-uniform (the reads below are
        // warp-collective)
        const bool ok = __syncthreads_and(mbar_wait(smem_u32(&mbar), phase));
        phase ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (!ok) {
            if (tid == 0) atomicExch(err, (int)DEV_TIMEOUT);
            mbar_wait(smem_u32(&mbar), phase ^ 1u);  // bounded: the MMAs may still be writing
            break;
        }
        {
            const int r = (warp & 3) * 32 + lane, half = warp >> 2, i = base + r;
            float acc[32];
            tc_ld32(tmem + ((unsigned)((warp & 3) * 32) << 16) + half * 32, acc);
            unsigned bits = 0u;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const float z = acc[j] + __ldg(&c[half * 32 + j]);
                if (z > 0.0f) bits |= 1u << j;
                acc[j] = z > 0.0f ? z : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < 32; j += 4)
                *reinterpret_cast<float4*>(&sZ[r * kZStride + half * 32 + j]) =
                    make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
            if (i < G.n) mask[2 * (size_t)i + half] = bits;
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int q = tid; q < kTcTile * 16; q += kTcThreads) {
            const int r = q >> 4, o = (q & 15) * 4, i = base + r;
            if (i >= G.n) continue;
            const float4 h = __ldg(reinterpret_cast<const float4*>(&Hin[(size_t)i * MH + o]));
            const float4 z = *reinterpret_cast<const float4*>(&sZ[r * kZStride + o]);
            *reinterpret_cast<float4*>(&Hout[(size_t)i * MH + o]) =
                make_float4(h.x + z.x, h.y + z.y, h.z + z.z, h.w + z.w);
        }
        __syncthreads();  // sZ is free for the next tile's operands
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) tc_dealloc(tmem_slot, MH);
}

// Backward node part on tcgen05: [dself ; dm] = dz W for tiles of 128 nodes (M = 128, N = 128
// inputs, K = 64 outputs in four MMAs); dz = dh * mask; writes dh + dself and dm / d_i.  Bound by
// traffic (rows of dh read twice, two rows written).  Measured at 499,288 nodes: 682 us with a
// row per thread in the epilogue (32 rows per store) -> 105 us.
constexpr int kTcBnSmem = kTcRegionZ + MK * MH * 2;
__global__ void __launch_bounds__(kTcThreads, kTcCtasPerSm) k_mpnn_layer_back_nodes_tc(
    Graph G, const float* __restrict__ dH, const unsigned* __restrict__ mask, const __nv_bfloat16* __restrict__ Wb,
    float* dSelf, float* dMs, int* err) {
    extern __shared__ __align__(1024) unsigned char tc_smem[];
    unsigned char* sA = tc_smem;                     // dz [node][out]
    float* sZ = reinterpret_cast<float*>(tc_smem);   // results, 64 columns at a time
    unsigned char* sB = tc_smem + kTcRegionZ;        // W^T [in][out]
    __shared__ __align__(8) unsigned long long mbar;
    __shared__ unsigned tmem_slot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) tc_alloc(&tmem_slot, MK);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar)));
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    for (int q = tid; q < MH * MK; q += kTcThreads) {
        const int o = q / MK, k = q % MK;
        *reinterpret_cast<__nv_bfloat16*>(sB + tc_offset(k, o, MK)) = Wb[q];
    }
    const int ntiles = (G.n + kTcTile - 1) / kTcTile;
    unsigned phase = 0;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int base = tile * kTcTile;
        for (int q = tid; q < kTcTile * 16; q += kTcThreads) {
            const int r = q >> 4, o = (q & 15) * 4, i = base + r;
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (i < G.n) {
                const unsigned b = __ldg(&mask[2 * (size_t)i + (o >> 5)]) >> (o & 31);
                v = __ldg(reinterpret_cast<const float4*>(&dH[(size_t)i * MH + o]));
                v = make_float4(b & 1u ? v.x : 0.0f, b & 2u ? v.y : 0.0f, b & 4u ? v.z : 0.0f, b & 8u ? v.w : 0.0f);
            }
            *reinterpret_cast<uint2*>(sA + tc_offset(r, o, kTcTile)) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
        }
        tc_sync_in();
        const unsigned tmem = tmem_slot;
        if (tid == 0) {
            const unsigned a0 = smem_u32(sA), b0 = smem_u32(sB);
            constexpr unsigned idesc = tc_idesc(kTcTile, MK);
#pragma unroll
            for (int ks = 0; ks < MH / 16; ++ks)
                tc_mma(tmem, tc_desc(a0 + ks * 2 * (kTcTile * 16), kTcTile * 16, 128),
                       tc_desc(b0 + ks * 2 * (MK * 16), MK * 16, 128), idesc, ks > 0);
            tc_commit(smem_u32(&mbar));
        }
        const bool ok = __syncthreads_and(mbar_wait(smem_u32(&mbar), phase));
        phase ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (!ok) {
            if (tid == 0) atomicExch(err, (int)DEV_TIMEOUT);
            mbar_wait(smem_u32(&mbar), phase ^ 1u);
            break;
        }
#pragma unroll 1
        for (int p = 0; p < 2; ++p) {  // columns 64 p .. 64 p + 63: dself, then dm
            const int rr = (warp & 3) * 32 + lane, half = warp >> 2;
            float acc[32];
            tc_ld32(tmem + ((unsigned)((warp & 3) * 32) << 16) + p * MH + half * 32, acc);
#pragma unroll
            for (int j = 0; j < 32; j += 4)
                *reinterpret_cast<float4*>(&sZ[rr * kZStride + half * 32 + j]) =
                    make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncthreads();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int q = tid; q < kTcTile * 16; q += kTcThreads) {
                const int r = q >> 4, o = (q & 15) * 4, i = base + r;
                if (i >= G.n) continue;
                const float4 z = *reinterpret_cast<const float4*>(&sZ[r * kZStride + o]);
                if (p == 0) {
                    const float4 h = __ldg(reinterpret_cast<const float4*>(&dH[(size_t)i * MH + o]));
                    *reinterpret_cast<float4*>(&dSelf[(size_t)i * MH + o]) =
                        make_float4(h.x + z.x, h.y + z.y, h.z + z.z, h.w + z.w);
                } else {
                    const float d = __ldg(&G.deg_inv[i]);
                    *reinterpret_cast<float4*>(&dMs[(size_t)i * MH + o]) =
                        make_float4(z.x * d, z.y * d, z.z * d, z.w * d);
                }
            }
            __syncthreads();
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) tc_dealloc(tmem_slot, MK);
}

// Backward weight part on tcgen05: per-CTA partial dW[out][in] = sum over the CTA's node
// tiles of [h ; m]^T dz (M = 128 inputs, N = 64 outputs, K = 128 nodes per tile,
// accumulated in tensor memory across the tiles) and dc on the CUDA cores.  A thread packs eight
// nodes of one feature into the 16 bytes they take in the K-major operand (coalesced loads, no
// bank conflicts); a tile's operands are overwritten only after its MMAs completed (mbarrier
// phase per tile).  Bound by DRAM traffic (rows of h, m and dh).  Measured at 499,288 nodes: 626 us
// with 2-byte stores and dc summed by 64 threads -> 137 us.
__global__ void __launch_bounds__(kTcThreads, 2) k_mpnn_layer_back_weights_tc(
    Graph G, const float* __restrict__ Hin, const float* __restrict__ M, const float* __restrict__ dH,
    const unsigned* __restrict__ mask, float* part, int* err) {
    extern __shared__ __align__(1024) unsigned char tc_smem[];
    unsigned char* sA = tc_smem;                      // [h ; m]^T [in][node]
    unsigned char* sB = tc_smem + MK * kTcTile * 2;   // dz^T [out][node]
    __shared__ __align__(8) unsigned long long mbar;
    __shared__ unsigned tmem_slot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) tc_alloc(&tmem_slot, MH);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar)));
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    const int ntiles = (G.n + kTcTile - 1) / kTcTile;
    const int o = tid & (MH - 1);
    unsigned phase = 0;
    bool ok = true, issued = false;
    float dc = 0.0f;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int base = tile * kTcTile;
        for (int rb = tid >> 6; rb < kTcTile / 8; rb += kTcThreads / MH) {
            float h[8], m[8], z[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int i = base + rb * 8 + u;
                const bool in = i < G.n;
                const size_t e = (size_t)i * MH + o;
                h[u] = in ? __ldg(&Hin[e]) : 0.0f;
                m[u] = in ? __ldg(&M[e]) : 0.0f;
                z[u] = in && ((__ldg(&mask[2 * (size_t)i + (o >> 5)]) >> (o & 31)) & 1u) ? __ldg(&dH[e]) : 0.0f;
            }
            if (issued && rb == (tid >> 6)) {  // the previous tile's MMAs have read the operands
                ok = __syncthreads_and(mbar_wait(smem_u32(&mbar), phase));
                phase ^= 1u;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (!ok) break;
            }
            auto pack = [](const float* v) {
                return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
            };
            *reinterpret_cast<uint4*>(sA + tc_offset(o, rb * 8, MK)) = pack(h);
            *reinterpret_cast<uint4*>(sA + tc_offset(MH + o, rb * 8, MK)) = pack(m);
            *reinterpret_cast<uint4*>(sB + tc_offset(o, rb * 8, MH)) = pack(z);
        }
        if (!ok) break;
        tc_sync_in();
        if (tid == 0) {
            const unsigned a0 = smem_u32(sA), b0 = smem_u32(sB);
            constexpr unsigned idesc = tc_idesc(MK, MH);
#pragma unroll
            for (int ks = 0; ks < kTcTile / 16; ++ks)
                tc_mma(tmem_slot, tc_desc(a0 + ks * 2 * (MK * 16), MK * 16, 128),
                       tc_desc(b0 + ks * 2 * (MH * 16), MH * 16, 128), idesc, (issued || ks > 0) ? 1 : 0);
            tc_commit(smem_u32(&mbar));
        }
        // dc: the outputs' sums of the rounded dz over the tile's nodes in order, beside the MMAs
        if (tid >= kTcThreads - MH) {
            float s = 0.0f;
#pragma unroll 4
            for (int rb = 0; rb < kTcTile / 8; ++rb) {
                const uint4 v = *reinterpret_cast<const uint4*>(sB + tc_offset(o, rb * 8, MH));
                const unsigned w[4] = { v.x, v.y, v.z, v.w };
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    s += __uint_as_float(w[u] << 16);
                    s += __uint_as_float(w[u] & 0xffff0000u);
                }
            }
            dc += s;
        }
        issued = true;
    }
    if (issued && ok) {
        ok = __syncthreads_and(mbar_wait(smem_u32(&mbar), phase));
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    if (!ok) {
        if (tid == 0) atomicExch(err, (int)DEV_TIMEOUT);
        if (issued) mbar_wait(smem_u32(&mbar), phase);
    }
    float* P = part + (size_t)blockIdx.x * (MH * MK + MH);
    const unsigned tmem = tmem_slot;
    const int in = (warp & 3) * 32 + lane, q = warp >> 2;  // accumulator lane = input row of dW^T
    float acc[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) acc[j] = 0.0f;
    if (issued && ok) tc_ld32(tmem + ((unsigned)((warp & 3) * 32) << 16) + q * 32, acc);
#pragma unroll
    for (int j = 0; j < 32; ++j) P[(q * 32 + j) * MK + in] = acc[j];
    if (tid >= kTcThreads - MH) P[MH * MK + o] = dc;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) tc_dealloc(tmem_slot, MH);
}

// y = w4 . h + c4 (terms in feature order) for tiles of 128 nodes whose rows are staged in shared
// memory by coalesced loads.  With a target also the backward pass of the output layer: dy =
// 2 (y - t) / n, dh = dy w4, and per-CTA partials of (dw4, dc4) and of the loss.  Bound by traffic (one
// row read, one written).  Measured at 499,288 nodes, training: 116 us for y and 302 us for the
// gradients as two kernels with a thread per node -> 46 us.
constexpr int kDecThreads = 256;
constexpr int kDecTile = 128;
constexpr int kDecStride = MH + 1;
__global__ void __launch_bounds__(kDecThreads) k_mpnn_decoder(int n, const float* __restrict__ H,
                                                              const float* __restrict__ P, float* y,
                                                              const float* __restrict__ target, float* dH,
                                                              double* part /* [grid][MH + 1] */, double* loss_part) {
    __shared__ float sH[kDecTile * kDecStride];
    __shared__ float sW[MH + 1], sD[kDecTile], sP[kDecThreads / MH][MH + 1];
    static_assert(kDecThreads / MH == 4 && kDecTile == 128, "32 nodes per partial sum, four per tile");
    __shared__ double sh[40];
    const int tid = threadIdx.x;
    if (tid <= MH) sW[tid] = P[kParamW4 + tid];  // w4, then c4
    const int o = tid & (MH - 1), g = tid >> 6;
    double grad = 0.0;  // threads 0 .. MH: (dw4, dc4) over this block's tiles
    double loss = 0.0;
    for (int base = blockIdx.x * kDecTile; base < n; base += gridDim.x * kDecTile) {
        __syncthreads();  // the previous tile's readers are done
        for (int q = tid; q < kDecTile * 16; q += kDecThreads) {
            const int r = q >> 4, f = (q & 15) * 4, i = base + r;
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (i < n) v = __ldg(reinterpret_cast<const float4*>(&H[(size_t)i * MH + f]));
            float* d = &sH[r * kDecStride + f];
            d[0] = v.x;
            d[1] = v.y;
            d[2] = v.z;
            d[3] = v.w;
        }
        __syncthreads();
        if (tid < kDecTile) {
            const int i = base + tid;
            float s = sW[MH];
#pragma unroll 16
            for (int k = 0; k < MH; ++k) s += sW[k] * sH[tid * kDecStride + k];
            float d = 0.0f;
            if (i < n) {
                y[i] = s;
                if (target) {
                    const float r = s - target[i];
                    d = 2.0f * r / (float)n;
                    loss += (double)r * r;
                }
            }
            sD[tid] = d;
        }
        if (!target) continue;
        __syncthreads();
        for (int q = tid; q < kDecTile * 16; q += kDecThreads) {
            const int r = q >> 4, f = (q & 15) * 4, i = base + r;
            if (i >= n) continue;
            const float d = sD[r];
            *reinterpret_cast<float4*>(&dH[(size_t)i * MH + f]) =
                make_float4(d * sW[f], d * sW[f + 1], d * sW[f + 2], d * sW[f + 3]);
        }
        // the tile's (dw4, dc4): 32 nodes by a binary tree (node l with l + 16, ...), the four sums in
        // order, the tiles in FP64
        auto tree = [&](auto term) {
            float v[16];
#pragma unroll
            for (int l = 0; l < 16; ++l) v[l] = __fadd_rn(term(l), term(l + 16));
#pragma unroll
            for (int d = 8; d > 0; d >>= 1)
#pragma unroll
                for (int l = 0; l < d; ++l) v[l] = __fadd_rn(v[l], v[l + d]);
            return v[0];
        };
        sP[g][o] = tree([&](int l) { return __fmul_rn(sD[32 * g + l], sH[(32 * g + l) * kDecStride + o]); });
        if (o == 0) sP[g][MH] = tree([&](int l) { return sD[32 * g + l]; });
        __syncthreads();
        if (tid <= MH) grad += (double)(((sP[0][tid] + sP[1][tid]) + sP[2][tid]) + sP[3][tid]);
    }
    if (!target) return;
    loss = block_sum(loss, sh);
    if (tid <= MH) part[(size_t)blockIdx.x * (MH + 1) + tid] = grad;
    if (tid == 0) loss_part[blockIdx.x] = loss;
}

// ---------------------------------------------------------------- backward
// One layer backward, node part: dz = dh * mask; [dself ; dm] = dz W (tensor cores);
// writes dself and dm / d_i.
__global__ void __launch_bounds__(kMpnnThreads) k_mpnn_layer_back_nodes(Graph G, const float* __restrict__ dH,
                                                                        const unsigned long long* __restrict__ mask,
                                                                        const __nv_bfloat16* __restrict__ Wb,
                                                                        float* dSelf, float* dMs) {
    __shared__ __align__(16) __nv_bfloat16 sZ[kTile][MH + kPad];
    __shared__ __align__(16) __nv_bfloat16 sWT[MK][MH + kPad];  // W^T: [in][out]
    const int base = blockIdx.x * kTile;
    for (int q = threadIdx.x; q < MH * MK; q += blockDim.x) {
        const int o = q / MK, k = q % MK;
        sWT[k][o] = Wb[q];
    }
    for (int q = threadIdx.x; q < kTile * MH; q += blockDim.x) {
        const int r = q / MH, o = q % MH, i = base + r;
        float v = 0.0f;
        if (i < G.n && ((mask[i] >> o) & 1ull)) v = dH[(size_t)i * MH + o];
        sZ[r][o] = __float2bfloat16_rn(v);
    }
    __syncthreads();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    float acc[MK / 8][4];
#pragma unroll
    for (int nt = 0; nt < MK / 8; ++nt)
        for (int k = 0; k < 4; ++k) acc[nt][k] = 0.0f;
    warp_gemm<MH / 16, MK / 8>(&sZ[w * 16][0], MH + kPad, &sWT[0][0], MH + kPad, acc);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int i = base + w * 16 + g + 8 * half;
        if (i >= G.n) continue;
        const float di = G.deg_inv[i];
#pragma unroll
        for (int nt = 0; nt < MK / 8; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int k = nt * 8 + 2 * t + e;
                const float v = acc[nt][2 * half + e];
                if (k < MH) dSelf[(size_t)i * MH + k] = v;
                else dMs[(size_t)i * MH + (k - MH)] = v * di;
            }
    }
}

// dh_prev_i = (dh_i + dself_i) + sum_{k in N(i)} dm_k / d_k (the graph is symmetric); dH null:
// dSelf holds dh + dself.  Measured at 499,288 nodes: 257 us with a thread per (node, feature) ->
// 91 us.
__global__ void __launch_bounds__(kRowThreads) k_mpnn_agg_back(Graph G, const float* __restrict__ dH,
                                                               const float* __restrict__ dSelf,
                                                               const float* __restrict__ dMs, float* dHprev) {
    const int i = blockIdx.x * kRowNodes + (threadIdx.x >> 4), o = (threadIdx.x & 15) * 4;
    if (i >= G.n) return;
    const size_t q = (size_t)i * MH + o;
    float4 s = __ldg(reinterpret_cast<const float4*>(&dSelf[q]));
    if (dH) {
        const float4 h = __ldg(reinterpret_cast<const float4*>(&dH[q]));
        s = make_float4(h.x + s.x, h.y + s.y, h.z + s.z, h.w + s.w);
    }
    *reinterpret_cast<float4*>(&dHprev[q]) = gather_rows(G, dMs, i, o, s);
}

// One layer backward, weight part: per-CTA partial dW (= [h ; m]^T dz, tensor cores) and
// dc, over the node tiles this CTA visits.
__global__ void __launch_bounds__(kMpnnThreads) k_mpnn_layer_back_weights(Graph G, const float* __restrict__ Hin,
                                                                          const float* __restrict__ M,
                                                                          const float* __restrict__ dH,
                                                                          const unsigned long long* __restrict__ mask,
                                                                          float* part /* [grid][MH*MK + MH] */) {
    __shared__ __align__(16) __nv_bfloat16 sAT[MK][kTile + kPad];  // [in][node]
    __shared__ __align__(16) __nv_bfloat16 sZT[MH][kTile + kPad];  // [out][node]
    __shared__ float sC[MH];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    // warp w owns rows (inputs) w*32 .. w*32+31: two m tiles
    float acc[2][MH / 8][4];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < MH / 8; ++nt)
            for (int k = 0; k < 4; ++k) acc[mt][nt][k] = 0.0f;
    for (int o = threadIdx.x; o < MH; o += blockDim.x) sC[o] = 0.0f;
    const int ntiles = (G.n + kTile - 1) / kTile;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int base = tile * kTile;
        __syncthreads();
        for (int q = threadIdx.x; q < kTile * MH; q += blockDim.x) {
            const int r = q / MH, o = q % MH, i = base + r;
            float h = 0.0f, m = 0.0f, z = 0.0f;
            if (i < G.n) {
                h = Hin[(size_t)i * MH + o];
                m = M[(size_t)i * MH + o];
                if ((mask[i] >> o) & 1ull) z = dH[(size_t)i * MH + o];
            }
            sAT[o][r] = __float2bfloat16_rn(h);
            sAT[MH + o][r] = __float2bfloat16_rn(m);
            sZT[o][r] = __float2bfloat16_rn(z);
        }
        __syncthreads();
        for (int o = threadIdx.x; o < MH; o += blockDim.x) {
            float s = 0.0f;
            for (int r = 0; r < kTile; ++r) s += __bfloat162float(sZT[o][r]);
            sC[o] += s;
        }
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
            warp_gemm<kTile / 16, MH / 8>(&sAT[w * 32 + mt * 16][0], kTile + kPad, &sZT[0][0], kTile + kPad, acc[mt]);
    }
    __syncthreads();
    // dW[out][in] = acc[in][out]
    float* P = part + (size_t)blockIdx.x * (MH * MK + MH);
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int in = w * 32 + mt * 16 + g + 8 * half;
#pragma unroll
            for (int nt = 0; nt < MH / 8; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int o = nt * 8 + 2 * t + e;
                    P[o * MK + in] = acc[mt][nt][2 * half + e];
                }
        }
    for (int o = threadIdx.x; o < MH; o += blockDim.x) P[MH * MK + o] = sC[o];
}

// Encoder backward: per-block partials of (dW0, dc0).  Thread (o, k) sums dz_o f_k (k < MIN) or
// dz_o (k == MIN) over the block's nodes in order, from tiles of 64 nodes staged in shared memory
// by coalesced loads, the next tile's loads in flight meanwhile.  Measured at 499,288 nodes:
// 1,800 us with every thread loading its own terms -> 116 us.
constexpr int kEncThreads = MH * (MIN + 1);
constexpr int kEncTile = 64;
__global__ void __launch_bounds__(kEncThreads) k_mpnn_encoder_back(int n, const float* __restrict__ feat,
                                                                   const float* __restrict__ dH,
                                                                   const unsigned* __restrict__ mask0,
                                                                   float* part /* [grid][MH*MIN+MH] */) {
    __shared__ __align__(16) float sD[kEncTile][MH];
    __shared__ float sF[kEncTile][MIN];
    __shared__ unsigned sM[kEncTile][2];
    const int tid = threadIdx.x, o = tid / (MIN + 1), k = tid % (MIN + 1);
    const int nper = (n + gridDim.x - 1) / gridDim.x;
    const int i0 = (int)std::min((long long)n, (long long)blockIdx.x * nper), i1 = min(n, i0 + nper);
    constexpr int V = (kEncTile * 16 + kEncThreads - 1) / kEncThreads;  // float4 of dz per thread
    float4 d[V];
    float f = 0.0f;
    unsigned m = 0u;
    auto load = [&](int base) {
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int q = tid + v * kEncThreads, i = base + (q >> 4);
            if (q < kEncTile * 16 && i < i1) d[v] = __ldg(reinterpret_cast<const float4*>(&dH[(size_t)i * MH + (q & 15) * 4]));
        }
        if (tid < kEncTile * MIN && base + tid / MIN < i1) f = __ldg(&feat[(size_t)base * MIN + tid]);
        if (tid < 2 * kEncTile && base + tid / 2 < i1) m = __ldg(&mask0[2 * (size_t)base + tid]);
    };
    static_assert(kEncTile * MIN <= kEncThreads && 2 * kEncTile <= kEncThreads, "one feature and mask word per thread");
    float s = 0.0f;
    if (i0 < i1) load(i0);
    for (int base = i0; base < i1; base += kEncTile) {
        __syncthreads();  // the previous tile's readers are done
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int q = tid + v * kEncThreads;
            if (q < kEncTile * 16) *reinterpret_cast<float4*>(&sD[q >> 4][(q & 15) * 4]) = d[v];
        }
        if (tid < kEncTile * MIN) (&sF[0][0])[tid] = f;
        if (tid < 2 * kEncTile) (&sM[0][0])[tid] = m;
        __syncthreads();
        if (base + kEncTile < i1) load(base + kEncTile);
        const int cnt = min(kEncTile, i1 - base);
        for (int r = 0; r < cnt; ++r) {
            if (!((sM[r][o >> 5] >> (o & 31)) & 1u)) continue;
            const float dz = sD[r][o];
            s += (k < MIN) ? dz * sF[r][k < MIN ? k : 0] : dz;
        }
    }
    float* P = part + (size_t)blockIdx.x * (MH * MIN + MH);
    if (k < MIN) P[o * MIN + k] = s;
    else P[MH * MIN + o] = s;
}

// grad[off + j] = sum_b part[b * width + j], fixed order, FP64 accumulation: a block takes 32
// columns, warp w the rows w, w + 8, ...; the eight sums are added in order.
template <class T>
__global__ void __launch_bounds__(256) k_reduce_cols(const T* __restrict__ part, int nb, int width, float* grad, int off) {
    __shared__ double sh[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int j = blockIdx.x * 32 + lane;
    double s = 0.0;
    if (j < width) {
#pragma unroll 4
        for (int b = w; b < nb; b += 8) s += (double)__ldg(&part[(size_t)b * width + j]);
    }
    sh[w][lane] = s;
    __syncthreads();
    if (w == 0 && j < width) {
#pragma unroll
        for (int k = 1; k < 8; ++k) s += sh[k][lane];
        grad[off + j] = (float)s;
    }
}

__global__ void k_adamw(int np, float* P, const float* __restrict__ g, float* m, float* v, float c1, float c2,
                        float lr, float b1, float b2, float eps, float wd) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= np) return;
    const float gk = g[k];
    const float mk = b1 * m[k] + (1.0f - b1) * gk;
    const float vk = b2 * v[k] + (1.0f - b2) * gk * gk;
    m[k] = mk;
    v[k] = vk;
    P[k] -= lr * (mk / c1 / (sqrtf(vk / c2) + eps) + wd * P[k]);
}

__global__ void k_weights_bf16(const float* __restrict__ P, __nv_bfloat16* Wb) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= ML * MH * MK) return;
    const int l = q / (MH * MK), r = q % (MH * MK);
    Wb[q] = __float2bfloat16_rn(P[kParamLayer0 + l * kLayerSize + r]);
}

__global__ void k_deg_inv(int n, const int* __restrict__ rowptr, const int* __restrict__ col, float* dinv) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int d = 0;
    for (int k = rowptr[i]; k < rowptr[i + 1]; ++k) d += (col[k] != i);
    dinv[i] = d ? 1.0f / (float)d : 0.0f;
}

}  // namespace pf2

using namespace pf2;

struct pf2_mpnn {
    int n = 0;
    const pf2_mesh* mesh = nullptr;
    DevBuf<float> P, grad, am, av, dinv, feat, y, H, M, dH, dH2, dSelf, dMs, part, target;
    DevBuf<unsigned long long> mask;
    DevBuf<__nv_bfloat16> Wb;
    DevBuf<double> loss_part, dpart;
    DevBuf<int> err;  // a tcgen05 wait that ran out (DEV_TIMEOUT)
    int step = 0;
    int wgrid = 0;  // blocks of the gradient kernels (rows of part)
    int tgrid = 0;  // persistent blocks of the layer kernels
    int dgrid = 0;  // blocks of the decoder (rows of dpart and loss_part)
    bool tc = true;  // the layer GEMMs on tcgen05 (PF2_MPNN_MMA=sync: mma.sync)
    Graph graph() const { return Graph{ n, mesh->rowptr.p, mesh->col.p, dinv.p }; }
    float* Hl(int l) { return H.p + (size_t)l * n * MH; }
    float* Ml(int l) { return M.p + (size_t)l * n * MH; }
    unsigned long long* maskl(int l) { return mask.p + (size_t)l * n; }
};

namespace pf2 {

// Sections: the parameter count, the FP32 parameters, the AdamW moments and step count.
// The BF16 weight copies follow from the parameters and are rebuilt on reading.
pf2_status mpnn_checkpoint(pf2_mpnn* N, CkptFile& io, cudaStream_t st) {
    int meta[2] = { kParams, N->step };
    PF2_TRY(io.host("nmeta", meta, sizeof(meta)));
    PF2_REQUIRE(meta[0] == kParams, PF2_BAD_INPUT, "checkpoint network has %d parameters, this one %d", meta[0],
                kParams);
    PF2_TRY(io.device("nparams", N->P.p, sizeof(float) * kParams, st));
    PF2_TRY(io.device("nadam_m", N->am.p, sizeof(float) * kParams, st));
    PF2_TRY(io.device("nadam_v", N->av.p, sizeof(float) * kParams, st));
    if (!io.writing()) {
        N->step = meta[1];
        k_weights_bf16<<<blocks_for(ML * MH * MK), kThreads, 0, st>>>(N->P.p, N->Wb.p);
        PF2_LAUNCH_CHECK();
        PF2_CUDA(cudaStreamSynchronize(st));
    }
    return PF2_OK;
}

static unsigned* words(unsigned long long* m) { return reinterpret_cast<unsigned*>(m); }

static pf2_status mpnn_forward(pf2_mpnn* N, cudaStream_t st) {
    const Graph G = N->graph();
    k_mpnn_encoder<<<std::min(blocks_for(N->n, kRowNodes), (unsigned)num_sms() * 8), kRowThreads, 0, st>>>(
        G, N->feat.p, N->P.p, N->Hl(0), N->maskl(0));
    PF2_LAUNCH_CHECK();
    const unsigned tiles = blocks_for(N->n, kTile);
    for (int l = 0; l < ML; ++l) {
        if (N->tc)
            k_mpnn_layer_tc<<<N->tgrid, kTcThreads, kTcSmem, st>>>(
                G, N->Hl(l), N->Wb.p + (size_t)l * MH * MK, N->P.p + kParamLayer0 + l * kLayerSize + MH * MK,
                N->Hl(l + 1), N->Ml(l), words(N->maskl(l + 1)), N->err.p);
        else
            k_mpnn_layer<<<tiles, kMpnnThreads, 0, st>>>(G, N->Hl(l), N->Wb.p + (size_t)l * MH * MK,
                                                         N->P.p + kParamLayer0 + l * kLayerSize + MH * MK,
                                                         N->Hl(l + 1), N->Ml(l), N->maskl(l + 1));
        PF2_LAUNCH_CHECK();
    }
    return PF2_OK;
}

static pf2_status mpnn_decoder(pf2_mpnn* N, float* y, const float* target, cudaStream_t st) {
    k_mpnn_decoder<<<N->dgrid, kDecThreads, 0, st>>>(N->n, N->Hl(ML), N->P.p, y, target, target ? N->dH.p : nullptr,
                                                     target ? N->dpart.p : nullptr, target ? N->loss_part.p : nullptr);
    PF2_LAUNCH_CHECK();
    return PF2_OK;
}

template <class T>
static pf2_status reduce_cols(pf2_mpnn* N, const T* part, int nb, int width, int off, cudaStream_t st) {
    k_reduce_cols<T><<<blocks_for(width, 32), 256, 0, st>>>(part, nb, width, N->grad.p, off);
    PF2_LAUNCH_CHECK();
    return PF2_OK;
}

// After mpnn_decoder with a target: dH holds the gradient of the last layer's output, part the
// output layer's partials.
static pf2_status mpnn_backward(pf2_mpnn* N, cudaStream_t st) {
    const Graph G = N->graph();
    PF2_TRY(reduce_cols(N, N->dpart.p, N->dgrid, MH + 1, kParamW4, st));
    const unsigned tiles = blocks_for(N->n, kTile);
    float* dh = N->dH.p;
    float* dh2 = N->dH2.p;
    for (int l = ML - 1; l >= 0; --l) {
        const __nv_bfloat16* W = N->Wb.p + (size_t)l * MH * MK;
        if (N->tc)
            k_mpnn_layer_back_weights_tc<<<N->wgrid, kTcThreads, kTcBwSmem, st>>>(
                G, N->Hl(l), N->Ml(l), dh, words(N->maskl(l + 1)), N->part.p, N->err.p);
        else
            k_mpnn_layer_back_weights<<<N->wgrid, kMpnnThreads, 0, st>>>(G, N->Hl(l), N->Ml(l), dh,
                                                                         N->maskl(l + 1), N->part.p);
        PF2_LAUNCH_CHECK();
        PF2_TRY(reduce_cols(N, N->part.p, N->wgrid, kLayerSize, kParamLayer0 + l * kLayerSize, st));
        if (N->tc)
            k_mpnn_layer_back_nodes_tc<<<N->tgrid, kTcThreads, kTcBnSmem, st>>>(
                G, dh, words(N->maskl(l + 1)), W, N->dSelf.p, N->dMs.p, N->err.p);
        else
            k_mpnn_layer_back_nodes<<<tiles, kMpnnThreads, 0, st>>>(G, dh, N->maskl(l + 1), W, N->dSelf.p,
                                                                    N->dMs.p);
        PF2_LAUNCH_CHECK();
        k_mpnn_agg_back<<<blocks_for(N->n, kRowNodes), kRowThreads, 0, st>>>(G, N->tc ? nullptr : dh, N->dSelf.p,
                                                                             N->dMs.p, dh2);
        PF2_LAUNCH_CHECK();
        std::swap(dh, dh2);
    }
    k_mpnn_encoder_back<<<N->wgrid, kEncThreads, 0, st>>>(N->n, N->feat.p, dh, words(N->maskl(0)), N->part.p);
    PF2_LAUNCH_CHECK();
    return reduce_cols(N, N->part.p, N->wgrid, MH * MIN + MH, kParamW0, st);
}

}  // namespace pf2

extern "C" {

pf2_status pf2_mpnn_create(const pf2_mesh* mesh, unsigned long long seed, pf2_mpnn** out) {
    PF2_REQUIRE(mesh && out, PF2_BAD_INPUT, "null argument");
    *out = nullptr;
    pf2_mpnn* N = new pf2_mpnn();
    N->mesh = mesh;
    N->n = mesh->nv;
    const size_t n = N->n;
    auto fail = [&](pf2_status s) { delete N; return s; };
    N->wgrid = std::max(1, std::min((int)blocks_for(N->n, kTile), num_sms() * 2));
    N->tgrid = std::max(1, std::min((int)blocks_for(N->n, kTcTile), num_sms() * kTcCtasPerSm));
    N->dgrid = std::max(1, std::min((int)blocks_for(N->n, kDecTile), num_sms() * 4));
    const size_t part = (size_t)N->wgrid * (MH * MK + MH);
    pf2_status s;
    if ((s = N->P.alloc(kParams)) || (s = N->grad.alloc(kParams)) || (s = N->am.alloc(kParams)) ||
        (s = N->av.alloc(kParams)) || (s = N->dinv.alloc(n)) || (s = N->feat.alloc(n * MIN)) ||
        (s = N->y.alloc(n)) || (s = N->target.alloc(n)) ||
        (s = N->H.alloc((ML + 1) * n * MH)) || (s = N->M.alloc(ML * n * MH)) || (s = N->dH.alloc(n * MH)) ||
        (s = N->dH2.alloc(n * MH)) || (s = N->dSelf.alloc(n * MH)) || (s = N->dMs.alloc(n * MH)) ||
        (s = N->part.alloc(part)) || (s = N->mask.alloc((ML + 1) * n)) || (s = N->Wb.alloc(ML * MH * MK)) ||
        (s = N->loss_part.alloc(N->dgrid)) ||
        (s = N->dpart.alloc((size_t)N->dgrid * (MH + 1))) || (s = N->err.alloc(1)))
        return fail(s);
    if (const char* e = getenv("PF2_MPNN_MMA")) N->tc = strcmp(e, "sync") != 0;
    if (cudaMemset(N->err.p, 0, sizeof(int)) != cudaSuccess ||
        cudaFuncSetAttribute((void*)k_mpnn_layer_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem) !=
            cudaSuccess ||
        cudaFuncSetAttribute((void*)k_mpnn_layer_back_nodes_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kTcBnSmem) != cudaSuccess ||
        cudaFuncSetAttribute((void*)k_mpnn_layer_back_weights_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kTcBwSmem) != cudaSuccess)
        return fail(cuda_fail(cudaGetLastError(), "mpnn set-up", __FILE__, __LINE__));
    // He-style initialisation from a splitmix64 stream (deterministic for a seed);
    // the output layer starts at zero so the untrained guess is the extrapolation alone
    std::vector<float> h(kParams, 0.0f);
    unsigned long long st = seed;
    auto next = [&]() {
        st += 0x9E3779B97F4A7C15ull;
        unsigned long long z = st;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return (double)(z >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0;
    };
    for (int k = 0; k < MH * MIN; ++k) h[kParamW0 + k] = (float)(next() * std::sqrt(6.0 / MIN));
    for (int l = 0; l < ML; ++l)
        for (int k = 0; k < MH * MK; ++k)
            h[kParamLayer0 + l * kLayerSize + k] = (float)(next() * std::sqrt(6.0 / MK) * 0.5);
    if (cudaMemcpy(N->P.p, h.data(), sizeof(float) * kParams, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(N->am.p, 0, sizeof(float) * kParams) != cudaSuccess ||
        cudaMemset(N->av.p, 0, sizeof(float) * kParams) != cudaSuccess)
        return fail(cuda_fail(cudaGetLastError(), "mpnn init", __FILE__, __LINE__));
    k_deg_inv<<<blocks_for(N->n), kThreads>>>(N->n, mesh->rowptr.p, mesh->col.p, N->dinv.p);
    k_weights_bf16<<<blocks_for(ML * MH * MK), kThreads>>>(N->P.p, N->Wb.p);
    if (cudaDeviceSynchronize() != cudaSuccess) return fail(cuda_fail(cudaGetLastError(), "mpnn init", __FILE__, __LINE__));
    *out = N;
    return PF2_OK;
}

pf2_status pf2_mpnn_destroy(pf2_mpnn* N) {
    delete N;
    return PF2_OK;
}

int pf2_mpnn_param_count(void) { return kParams; }

pf2_status pf2_mpnn_save(const pf2_mpnn* N, const char* path) {
    PF2_REQUIRE(N && path, PF2_BAD_INPUT, "null argument");
    CkptFile io;
    PF2_TRY(io.open_write(path, CKPT_MPNN));
    PF2_TRY(mpnn_checkpoint(const_cast<pf2_mpnn*>(N), io, nullptr));
    return io.close();
}

pf2_status pf2_mpnn_load(pf2_mpnn* N, const char* path) {
    PF2_REQUIRE(N && path, PF2_BAD_INPUT, "null argument");
    CkptFile io;
    PF2_TRY(io.open_read(path, CKPT_MPNN));
    PF2_TRY(mpnn_checkpoint(N, io, nullptr));
    return io.close();
}

pf2_status pf2_mpnn_set_params(pf2_mpnn* N, const float* params_host) {
    PF2_REQUIRE(N && params_host, PF2_BAD_INPUT, "null argument");
    PF2_CUDA(cudaMemcpy(N->P.p, params_host, sizeof(float) * kParams, cudaMemcpyHostToDevice));
    k_weights_bf16<<<blocks_for(ML * MH * MK), kThreads>>>(N->P.p, N->Wb.p);
    PF2_LAUNCH_CHECK();
    PF2_CUDA(cudaDeviceSynchronize());
    return PF2_OK;
}

pf2_status pf2_mpnn_get_params(const pf2_mpnn* N, float* params_host, float* grad_host) {
    PF2_REQUIRE(N, PF2_BAD_INPUT, "null argument");
    PF2_CUDA(cudaDeviceSynchronize());
    int e = 0;
    PF2_CUDA(cudaMemcpy(&e, N->err.p, sizeof(int), cudaMemcpyDeviceToHost));
    PF2_REQUIRE(e == 0, (pf2_status)e, "a tensor-core wait timed out in the network's forward pass");
    if (params_host) PF2_CUDA(cudaMemcpy(params_host, N->P.p, sizeof(float) * kParams, cudaMemcpyDeviceToHost));
    if (grad_host) PF2_CUDA(cudaMemcpy(grad_host, N->grad.p, sizeof(float) * kParams, cudaMemcpyDeviceToHost));
    return PF2_OK;
}

pf2_status pf2_mpnn_forward(pf2_mpnn* N, const float* feat_dev, float* y_dev, void* stream) {
    PF2_REQUIRE(N && feat_dev && y_dev, PF2_BAD_INPUT, "null argument");
    cudaStream_t st = as_stream(stream);
    PF2_CUDA(cudaMemcpyAsync(N->feat.p, feat_dev, sizeof(float) * MIN * (size_t)N->n, cudaMemcpyDeviceToDevice, st));
    PF2_TRY(mpnn_forward(N, st));
    return mpnn_decoder(N, y_dev, nullptr, st);
}

pf2_status pf2_mpnn_train_step(pf2_mpnn* N, const float* feat_dev, const float* target_dev, float lr, int apply,
                               double* loss_host, void* stream) {
    PF2_REQUIRE(N && feat_dev && target_dev, PF2_BAD_INPUT, "null argument");
    cudaStream_t st = as_stream(stream);
    PF2_CUDA(cudaMemcpyAsync(N->feat.p, feat_dev, sizeof(float) * MIN * (size_t)N->n, cudaMemcpyDeviceToDevice, st));
    PF2_CUDA(cudaMemcpyAsync(N->target.p, target_dev, sizeof(float) * (size_t)N->n, cudaMemcpyDeviceToDevice, st));
    PF2_TRY(mpnn_forward(N, st));
    PF2_TRY(mpnn_decoder(N, N->y.p, N->target.p, st));
    PF2_TRY(mpnn_backward(N, st));
    if (apply) {
        ++N->step;
        const float b1 = 0.9f, b2 = 0.999f;
        const float c1 = 1.0f - std::pow(b1, (float)N->step), c2 = 1.0f - std::pow(b2, (float)N->step);
        k_adamw<<<blocks_for(kParams), kThreads, 0, st>>>(kParams, N->P.p, N->grad.p, N->am.p, N->av.p, c1, c2, lr,
                                                          b1, b2, 1e-8f, 0.01f);
        PF2_LAUNCH_CHECK();
        k_weights_bf16<<<blocks_for(ML * MH * MK), kThreads, 0, st>>>(N->P.p, N->Wb.p);
        PF2_LAUNCH_CHECK();
    }
    if (loss_host) {
        std::vector<double> lp(N->dgrid);
        PF2_CUDA(cudaMemcpyAsync(lp.data(), N->loss_part.p, sizeof(double) * lp.size(), cudaMemcpyDeviceToHost, st));
        PF2_CUDA(cudaStreamSynchronize(st));
        double s = 0.0;
        for (double v : lp) s += v;
        *loss_host = s / N->n;
    }
    return PF2_OK;
}

}  // extern "C"

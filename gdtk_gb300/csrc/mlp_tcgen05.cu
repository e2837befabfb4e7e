// mlp_tcgen05.cu -- the surrogate network on the fifth-generation tensor cores: a layer's forward GEMM (below), which
// training takes because it keeps every layer's activations, and inference of the whole network in one kernel
// (mlp_fused_kernel).
//
// The layer kernel:
//   D[M][N] = A[M][K] W[N][K]^T + bias, then GELU (keeping the pre-activation) or nothing,
// BF16 operands, FP32 accumulation in tensor memory (TMEM), K and N multiples of 16 up to 256.
//
// One persistent CTA per SM.  The CTA loads W once with TMA and keeps it in shared
// memory; for each 128-row tile of A it
//   1. loads the tile with TMA (2-D boxes of 8 elements x rows, which land as the K-major,
//      no-swizzle canonical layout: 8-row x 16-byte core matrices, rows 16 bytes apart, K-groups
//      rows x 16 bytes apart), completion counted in bytes on an mbarrier;
//   2. one thread issues K/16 tcgen05.mma (M = 128, N, K = 16) into an N-column FP32 accumulator
//      and tcgen05.commit arrives on a second mbarrier when they are done;
//   3. each warp reads its 32 TMEM lanes (= rows) with tcgen05.ld 32x32b, adds the bias, applies the
//      activation and stores FP32 and/or BF16 rows.
// Every mbarrier wait is bounded: on timeout the CTA records an error flag, waits (bounded) for
// what it has in flight, frees its TMEM and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <atomic>
#include <cstdlib>
#include <cstring>

#include "mlp_launch.h"

namespace gdtk {
namespace {

constexpr int TC_M = 128;                           // rows per tile = TMEM lanes
constexpr int EPI_WARPS = 16;                       // epilogue warps: 4 lane quarters x 4 column slices
constexpr int TC_THREADS = 32 * (1 + EPI_WARPS);
constexpr unsigned SPIN_LIMIT = 1u << 22;   // mbarrier polls before a wait gives up

__device__ int g_tc_error;

struct TcArgs {
    int M, N, K;
    int a_bytes, w_bytes;   // shared-memory bytes of one A tile and of W
    unsigned tmem_cols;
    const float* bias;
    int act;
    float* pre;
    float* D;
    __nv_bfloat16* Dh;
    int ldd;
};

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// Waits for the phase of parity `parity` to complete; false if it has not after SPIN_LIMIT polls.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity) {
    const unsigned a = smem_u32(bar);
    for (unsigned i = 0; i < SPIN_LIMIT; ++i) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor: start address, leading-dimension (K-direction) and stride-dimension
// (M/N-direction) byte offsets between core matrices, descriptor version 1, no swizzle.
__device__ __forceinline__ unsigned long long smem_desc(unsigned addr, unsigned lbo, unsigned sbo) {
    return (unsigned long long)((addr & 0x3FFFFu) >> 4) | (unsigned long long)((lbo >> 4) & 0x3FFFu) << 16 |
           (unsigned long long)((sbo >> 4) & 0x3FFFu) << 32 | 1ull << 46;
}

__device__ __forceinline__ void mma_bf16(unsigned tmem_d, unsigned long long adesc, unsigned long long bdesc,
                                         unsigned idesc, unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// Starts loading 16 consecutive FP32 columns of this thread's TMEM lane; the values are valid after
// tmem_ld_wait.
__device__ __forceinline__ void tmem_ld16(unsigned taddr, unsigned (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

// Waits for this thread's TMEM loads; the empty statements after it make every later use of r depend on
// the wait.
__device__ __forceinline__ void tmem_ld_wait(unsigned (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) asm volatile("" : "+r"(r[i])::"memory");
}
template <int Q>
__device__ __forceinline__ void tmem_ld_wait(unsigned (&r)[Q][16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
        for (int i = 0; i < 16; ++i) asm volatile("" : "+r"(r[q][i])::"memory");
}

// Two FP32 values in one 64-bit register, and the packed operations on them: one issue slot for two results.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float ex2_ftz(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rcp_ftz(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// GELU, tanh form, as the mma.sync kernel's epilogue, of two values: 0.5 x (1 + tanh(u)) = x / (1 + exp(-2u)),
// u = sqrt(2/pi) (x + 0.044715 x^3), with the 2-ulp exponential and reciprocal.  exp(-2u) -> inf gives -0, exp(-2u) -> 0
// gives x; flushing a subnormal exponential to zero or a reciprocal below 2^-126 changes neither.  The order of the
// operations is that of x + 0.044715f * x * x * x in FP32, to the bit: a last-place change here turns BF16 roundings.
__device__ __forceinline__ unsigned long long gelu2(unsigned long long x) {
    const float c1 = -2.0f * 0.7978845608028654f * 1.4426950408889634f, c3 = 0.044715f;
    const float2 d = unpack2(mul2(fma2(mul2(mul2(pack2(c3, c3), x), x), x, x), pack2(c1, c1)));
    const float2 w = unpack2(add2(pack2(ex2_ftz(d.x), ex2_ftz(d.y)), pack2(1.f, 1.f)));
    return mul2(x, pack2(rcp_ftz(w.x), rcp_ftz(w.y)));
}

__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Warp 0 (one lane) loads and issues the MMAs; warps 1..EPI_WARPS drain the accumulators.  Two TMEM
// accumulators alternate between tiles, so that the MMAs of tile i+1 (and the load of its A) run while
// the epilogue warps drain tile i.  Epilogue warp w reads TMEM lanes 32 (w % 4) .. + 31 (the lanes a warp
// may access) and the column slice (w - 1) / 4 of EPI_WARPS / 4 slices.
// Barriers: load (A tile, + W the first time), full[b] (tcgen05.commit of accumulator b), empty[b]
// (every epilogue warp has read accumulator b).
__global__ void __launch_bounds__(TC_THREADS, 1)
    gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, const TcArgs g) {
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* sA = smem;
    unsigned char* sW = smem + g.a_bytes;
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(smem + g.a_bytes + g.w_bytes);
    unsigned long long* bar_load = bars;
    unsigned long long* bar_full = bars + 1;    // [2]
    unsigned long long* bar_empty = bars + 3;   // [2]
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 5);
    int* s_state = reinterpret_cast<int*>(tmem_slot + 1);   // [0] failed, [1] commits issued
    float* s_bias = reinterpret_cast<float*>(bars + 8);       // [N]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = threadIdx.x; k < g.N; k += blockDim.x) s_bias[k] = g.bias ? g.bias[k] : 0.f;

    if (threadIdx.x == 0) {
        mbar_init(bar_load, 1);
        mbar_init(&bar_full[0], 1);
        mbar_init(&bar_full[1], 1);
        mbar_init(&bar_empty[0], EPI_WARPS);
        mbar_init(&bar_empty[1], EPI_WARPS);
        s_state[0] = 0;
        s_state[1] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(2 * g.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *tmem_slot;
    const int ntiles = (g.M + TC_M - 1) / TC_M;
    const int my_tiles = blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;

    if (warp == 0) {
        if (lane == 0) {
            // instruction descriptor: FP32 accumulator, BF16 A and B, both K-major, N >> 3, M >> 4
            const unsigned idesc =
                (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(g.N >> 3) << 17) | ((unsigned)(TC_M >> 4) << 24);
            const unsigned a_lbo = TC_M * 16, w_lbo = (unsigned)g.N * 16;   // bytes between K-groups
            const int kgroups = g.K / 8;
            int failed = 0, commits = 0;
            unsigned load_parity = 0;
            for (int i = 0; i < my_tiles && !failed; ++i) {
                const int tile = blockIdx.x + i * gridDim.x, b = i & 1;
                // A is free once the previous tile's MMAs are done (its commit)
                if (i > 0 && !mbar_wait(&bar_full[(i - 1) & 1], ((i - 1) >> 1) & 1)) { failed = 2; break; }
                mbar_expect_tx(bar_load, (unsigned)(g.a_bytes + (i == 0 ? g.w_bytes : 0)));
                for (int kg = 0; kg < kgroups; ++kg) tma_load_2d(sA + kg * a_lbo, &tmA, kg * 8, tile * TC_M, bar_load);
                if (i == 0)
                    for (int kg = 0; kg < kgroups; ++kg) tma_load_2d(sW + kg * w_lbo, &tmW, kg * 8, 0, bar_load);
                load_parity = i & 1;
                if (!mbar_wait(bar_load, load_parity)) { failed = 1; break; }
                // accumulator b is free once the epilogue has drained its previous tile
                if (i >= 2 && !mbar_wait(&bar_empty[b], ((i >> 1) - 1) & 1)) { failed = 3; break; }
                tc_fence_after();
                const unsigned acc = tmem + (unsigned)b * g.tmem_cols;
                for (int ks = 0; ks < g.K / 16; ++ks) {   // one K = 16 step covers two K-groups
                    const unsigned long long ad = smem_desc(smem_u32(sA) + 2u * ks * a_lbo, a_lbo, 128);
                    const unsigned long long bd = smem_desc(smem_u32(sW) + 2u * ks * w_lbo, w_lbo, 128);
                    mma_bf16(acc, ad, bd, idesc, ks > 0 ? 1u : 0u);
                }
                mma_commit(&bar_full[b]);
                ++commits;
            }
            s_state[1] = commits;
            if (failed) {
                atomicExch(&g_tc_error, failed);
                s_state[0] = 1;
                if (failed == 1) mbar_wait(bar_load, load_parity);   // bounded: the loads still in flight
            }
        }
    } else if (warp <= EPI_WARPS) {
        const int quarter = warp & 3, slice = (warp - 1) >> 2, slices = EPI_WARPS / 4;
        const int chunks = g.N / 16;   // 16-column chunks; this warp's are [slice, slice + 1) x chunks / slices
        const int c0 = 16 * (slice * chunks / slices), c1 = 16 * ((slice + 1) * chunks / slices);
        for (int i = 0; i < my_tiles; ++i) {
            const int tile = blockIdx.x + i * gridDim.x, b = i & 1;
            if (!mbar_wait(&bar_full[b], (i >> 1) & 1)) {
                if (lane == 0) atomicExch(&g_tc_error, 4);
                break;
            }
            tc_fence_after();
            const int row = tile * TC_M + quarter * 32 + lane;
            const unsigned trow = tmem + (unsigned)b * g.tmem_cols + ((unsigned)(quarter * 32) << 16);
            const int nq = (c1 - c0) >> 4;   // at most 4: N <= 256 over 4 column slices
            for (int qb = 0; qb < nq; qb += 2) {   // two 16-column chunks in flight per wait
                unsigned r[2][16];
                __syncwarp();   // the TMEM loads are warp-collective
                tmem_ld16(trow + (unsigned)(c0 + 16 * qb), r[0]);
                if (qb + 1 < nq) tmem_ld16(trow + (unsigned)(c0 + 16 * qb + 16), r[1]);
                tmem_ld_wait(r);
                if (row >= g.M) continue;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (qb + q >= nq) break;
                    const int c = c0 + 16 * (qb + q);
                    const size_t o = (size_t)row * g.ldd + c;
                    float v[16];
#pragma unroll
                    for (int k = 0; k < 16; k += 2) {
                        v[k] = __uint_as_float(r[q][k]) + s_bias[c + k];
                        v[k + 1] = __uint_as_float(r[q][k + 1]) + s_bias[c + k + 1];
                        if (g.act == ACT_GELU) {
                            if (g.pre) {
                                g.pre[o + k] = v[k];
                                g.pre[o + k + 1] = v[k + 1];
                            }
                            const float2 h = unpack2(gelu2(pack2(v[k], v[k + 1])));
                            v[k] = h.x;
                            v[k + 1] = h.y;
                        }
                    }
                    if (g.D) {
                        float4* d4 = reinterpret_cast<float4*>(g.D + o);
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            d4[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
                    }
                    if (g.Dh) {
                        __align__(16) __nv_bfloat16 h[16];
#pragma unroll
                        for (int k = 0; k < 16; ++k) h[k] = __float2bfloat16(v[k]);
                        uint4* d = reinterpret_cast<uint4*>(g.Dh + o);
                        d[0] = reinterpret_cast<const uint4*>(h)[0];
                        d[1] = reinterpret_cast<const uint4*>(h)[1];
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_empty[b]);
        }
    }
    __syncthreads();
    if (s_state[0] && threadIdx.x == 0 && s_state[1] > 0) {   // bounded wait for the last commit before freeing TMEM
        const int last = s_state[1] - 1;
        mbar_wait(&bar_full[last & 1], (last >> 1) & 1);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * g.tmem_cols)
                     : "memory");
}

// ------------------------------------------------------------------------------------------------------------
// The whole inference network in one kernel: a row's activations stay in shared memory and tensor memory from the
// first layer to the last, so that device memory sees the input and the output rows only.
//
// One persistent CTA per SM works on two 128-row tiles at a time.  Each of the two slots has an activation tile in
// shared memory (BF16, the K-major no-swizzle layout), an FP32 accumulator of up to 256 TMEM columns and eight
// epilogue warps (two per TMEM lane quarter, half of the columns each).  A slot's layer is: MMAs from its tile into
// its accumulator; then its warps read the accumulator, add the bias, apply GELU and write the next layer's tile over
// the one that the MMAs have finished with.  While one slot is in its epilogue the other's MMAs run.  The weights are
// too large to stay (393 KB for three 256 x 256 layers) and come again for each slot's layer, 64 columns of K at a time,
// through a ring of TMA stages of 128-byte rows (narrower rows load slower than the MMAs read).  Rows and columns past
// a matrix's edge arrive as zeros, so sizes that are multiples of 8 are padded to 16.
//
// 262,147 rows of 16 -> 4 x 256 -> 16: 420 -> 182 us (five layer kernels, input and output passes before); 2,000 rows:
// 27 us; 4 x 128: 105 us, 2 x 64: 47 us.  What bounds it is shared memory: a tile's 256 x 256 layer reads 64 KB of
// activations and 128 KB of weights for the MMAs and writes 128 KB and 64 KB, about 3,100 cycles of its 4,900; its
// exponentials and reciprocals take 3,100 more, which the other slot's MMAs hide in part.
//
// A wait that gives up ends the CTA's work: the error flag is set, the rows that are not done become NaN (the surrogate
// update sends such cells to the FP64 update), and what is in flight is waited for.  The rows are written out of line: in
// the kernel's own code they cost the layers 1% (182.2 and 181.2 us).
struct FusedArgs {
    int M, nlayers;
    int dims[FUSED_MAX_LAYERS + 1];          // nin_pad, width ..., nout_pad (multiples of 8)
    int a_bytes, stage_bytes, stages;
    unsigned tmem_cols;                      // per slot
    const float* bias[FUSED_MAX_LAYERS];
    const __nv_bfloat16* Xh;                 // input rows in BF16, or
    const float *X, *xs, *xd;                // raw rows: bf16((X - xs) / xd)
    float* out;                              // [M][nout_pad]: the output, or with ys: output * yd + ys
    const float *ys, *yd;
    unsigned go;                             // 0, for testing: everything as after waits that gave up
};
struct FusedMaps {
    CUtensorMap w[FUSED_MAX_LAYERS];
};

constexpr int FUSED_SLOT_WARPS = 8;
constexpr int FUSED_THREADS = 32 * (2 + 2 * FUSED_SLOT_WARPS);
constexpr int FUSED_KC = 64;                 // K columns per weight stage: one row of the 128-byte swizzle

__host__ __device__ constexpr int pad16(int n) { return (n + 15) & ~15; }

// K-major operand in the 128-byte swizzle: 8-row groups 1024 bytes apart
__device__ __forceinline__ unsigned long long smem_desc_sw128(unsigned addr) {
    return (unsigned long long)((addr & 0x3FFFFu) >> 4) | 1ull << 16 | (unsigned long long)(1024 >> 4) << 32 | 1ull << 46 |
           2ull << 61;
}

// Eight columns from c of this thread's row, packed to BF16, into the row's 16 bytes of K-group c / 8.
__device__ __forceinline__ void store_group(unsigned char* a, int row, int c, const unsigned long long* v) {
    __nv_bfloat162 h[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 f = unpack2(v[k]);
        h[k] = __floats2bfloat162_rn(f.x, f.y);
    }
    *reinterpret_cast<uint4*>(a + (c >> 3) * (TC_M * 16) + row * 16) = *reinterpret_cast<const uint4*>(h);
}

__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// Eight output columns from c, times yd plus ys when those are set
__device__ __forceinline__ void store_out(const FusedArgs& g, unsigned row, int c, int nout, const unsigned long long* v) {
    if (c >= nout) return;
    float f[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 x = unpack2(v[k]);
        f[2 * k] = x.x;
        f[2 * k + 1] = x.y;
    }
    if (g.ys) {
        float ys[8], yd[8];
        load8(g.ys + c, ys);
        load8(g.yd + c, yd);
#pragma unroll
        for (int k = 0; k < 8; ++k) f[k] = f[k] * yd[k] + ys[k];
    }
    float4* o = reinterpret_cast<float4*>(g.out + (size_t)row * nout + c);
    o[0] = make_float4(f[0], f[1], f[2], f[3]);
    o[1] = make_float4(f[4], f[5], f[6], f[7]);
}

// A warp's rows and columns of the CTA's tiles from number `j` on, every other one
__device__ __noinline__ void nan_rows(float* out, int M, int nout, int j, int tiles, int r, int half) {
    const int chunks = pad16(nout) / 16, c1 = 16 * ((half + 1) * chunks / 2);
    for (; j < tiles; j += 2) {
        const unsigned row = (blockIdx.x + j * gridDim.x) * TC_M + r;
        if (row < (unsigned)M)
            for (int c = 16 * (half * chunks / 2); c < c1 && c < nout; ++c)
                out[(size_t)row * nout + c] = __int_as_float(0x7fffffff);
    }
}

__global__ void __launch_bounds__(FUSED_THREADS, 1)
    mlp_fused_kernel(const __grid_constant__ FusedMaps maps, const __grid_constant__ FusedArgs g) {
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* sW = smem;                                        // [stages][stage_bytes], on swizzle atoms
    unsigned char* sA = sW + g.stages * g.stage_bytes;               // [2][a_bytes]
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(sA + 2 * g.a_bytes);
    unsigned long long* w_full = bars;                               // [FUSED_MAX_STAGES]: a stage has landed
    unsigned long long* w_empty = bars + FUSED_MAX_STAGES;           // [FUSED_MAX_STAGES]: its MMAs are done
    unsigned long long* a_ready = bars + 2 * FUSED_MAX_STAGES;       // [2]: the slot's tile is written, its accumulator read
    unsigned long long* acc_full = a_ready + 2;                      // [2]: the slot's layer is in its accumulator
    unsigned long long* drained = a_ready + 4;                       // every MMA issued is done
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(a_ready + 5);
    unsigned long long* bias_ready = a_ready + 6;                    // [2]: the slot's biases of the layer are written
    float* s_bias = reinterpret_cast<float*>(a_ready + 8);           // [2][256], zeros past a layer's end
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int k = 0; k < g.stages; ++k) {
            mbar_init(&w_full[k], 1);
            mbar_init(&w_empty[k], 1);
        }
        for (int k = 0; k < 2; ++k) {
            mbar_init(&a_ready[k], FUSED_SLOT_WARPS);
            mbar_init(&acc_full[k], 1);
            mbar_init(&bias_ready[k], FUSED_SLOT_WARPS);
        }
        mbar_init(drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(2 * g.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *tmem_slot;
    const int ntiles = (g.M - 1) / TC_M + 1;
    const int my_tiles = blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    // the swizzle is of shared addresses; the declaration asks for this alignment
    const bool go = (smem_u32(smem) & 1023u) == 0 && g.go != 0;
    if (!go && threadIdx.x == 0) atomicExch(&g_tc_error, 6);
    // tile j of this CTA is in slot j & 1; the layers of a pair of tiles alternate between the slots

    if (warp == 0 && lane == 0) {   // MMAs
        int stage = 0, failed = 0;
        unsigned wpar = 0, issued = 0;
        for (int j0 = 0; go && j0 < my_tiles && !failed; j0 += 2)
            for (int l = 0; l < g.nlayers && !failed; ++l)
                for (int s = 0; s < 2 && j0 + s < my_tiles && !failed; ++s) {
                    const unsigned seq = (unsigned)(j0 >> 1) * g.nlayers + l;
                    if (!mbar_wait(&a_ready[s], seq & 1)) { failed = 3; break; }
                    tc_fence_after();
                    const unsigned a = smem_u32(sA + s * g.a_bytes), acc = tmem + (unsigned)s * g.tmem_cols;
                    const int K = pad16(g.dims[l]);
                    // FP32 accumulator, BF16 A and B, both K-major, N >> 3, M >> 4
                    const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) |
                                           ((unsigned)(pad16(g.dims[l + 1]) >> 3) << 17) | ((unsigned)(TC_M >> 4) << 24);
                    for (int k0 = 0; k0 < K; k0 += FUSED_KC) {
                        if (!mbar_wait(&w_full[stage], wpar)) { failed = 1; break; }
                        tc_fence_after();
                        const unsigned w = smem_u32(sW + stage * g.stage_bytes);
                        for (int k = k0; k < min(K, k0 + FUSED_KC); k += 16)
                            mma_bf16(acc, smem_desc(a + (k >> 3) * (TC_M * 16), TC_M * 16, 128),
                                     smem_desc_sw128(w + 2 * (k - k0)), idesc, k > 0 ? 1u : 0u);
                        mma_commit(&w_empty[stage]);
                        issued = 1;
                        if (++stage == g.stages) { stage = 0; wpar ^= 1; }
                    }
                    if (!failed) mma_commit(&acc_full[s]);
                }
        if (issued) {   // bounded: nothing of this CTA is in flight when it frees its memory
            mma_commit(drained);
            if (!mbar_wait(drained, 0) && !failed) failed = 2;
        }
        if (failed) atomicExch(&g_tc_error, failed);
    } else if (warp == 1 && lane == 0) {   // weights
        int stage = 0, failed = 0;
        unsigned par = 1, loads = 0;   // a first wait on the phase before the first passes
        for (int j0 = 0; go && j0 < my_tiles && !failed; j0 += 2)
            for (int l = 0; l < g.nlayers && !failed; ++l)
                for (int s = 0; s < 2 && j0 + s < my_tiles && !failed; ++s)
                    for (int k0 = 0; k0 < pad16(g.dims[l]); k0 += FUSED_KC) {
                        if (!mbar_wait(&w_empty[stage], par)) { failed = 5; break; }
                        mbar_expect_tx(&w_full[stage], (unsigned)pad16(g.dims[l + 1]) * FUSED_KC * 2);
                        tma_load_2d(sW + stage * g.stage_bytes, &maps.w[l], k0, 0, &w_full[stage]);
                        ++loads;
                        if (++stage == g.stages) { stage = 0; par ^= 1; }
                    }
        if (failed) atomicExch(&g_tc_error, failed);
        // bounded: the loads in flight, also where it is the MMAs' thread that gave up
        for (unsigned q = loads > (unsigned)g.stages ? loads - g.stages : 0; q < loads; ++q)
            mbar_wait(&w_full[q % g.stages], (q / g.stages) & 1);
    } else if (warp >= 2) {
        const int s = (warp - 2) / FUSED_SLOT_WARPS, half = ((warp - 2) % FUSED_SLOT_WARPS) >> 2;
        const int r = (warp & 3) * 32 + lane;   // the TMEM lanes that a warp may read are those of its number mod 4
        const int tid = (threadIdx.x - 64) & (32 * FUSED_SLOT_WARPS - 1);
        unsigned char* a = sA + s * g.a_bytes;
        float* bias = s_bias + s * 256;
        const unsigned trow = tmem + (unsigned)s * g.tmem_cols + ((unsigned)((warp & 3) * 32) << 16);
        const int nin = g.dims[0], nout = g.dims[g.nlayers];
        unsigned seq = 0;
        bool ok = go;
        int undone = ok ? my_tiles : s;   // the slot's first tile that is not done
        for (int j = s; j < my_tiles && ok; j += 2) {
            const unsigned row = (blockIdx.x + j * gridDim.x) * TC_M + r, M = g.M;
            // the input tile: the two warps of a lane quarter take every other K-group
            for (int c = 8 * half; c < pad16(nin); c += 16) {
                uint4 h = make_uint4(0u, 0u, 0u, 0u);
                if (row < M && c < nin) {
                    if (g.Xh) {
                        h = __ldg(reinterpret_cast<const uint4*>(g.Xh + (size_t)row * nin + c));
                    } else {
                        float x[8], m[8], d[8];
                        load8(g.X + (size_t)row * nin + c, x);
                        load8(g.xs + c, m);
                        load8(g.xd + c, d);
                        __nv_bfloat16 e[8];
#pragma unroll
                        for (int k = 0; k < 8; ++k) e[k] = __float2bfloat16((x[k] - m[k]) / d[k]);
                        memcpy(&h, e, 16);
                    }
                }
                *reinterpret_cast<uint4*>(a + (c >> 3) * (TC_M * 16) + r * 16) = h;
            }
            for (int l = 0; l < g.nlayers; ++l, ++seq) {
                const float b0 = tid < g.dims[l + 1] ? __ldg(g.bias[l] + tid) : 0.f;   // one column's bias per thread
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the tile, to the MMAs
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&a_ready[s]);
                // the accumulator; and every warp of the slot is done with the layer before
                ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[s], seq & 1));
                if (ok) {
                    bias[tid] = b0;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bias_ready[s]);
                    ok = __all_sync(0xffffffffu, mbar_wait(&bias_ready[s], seq & 1));
                }
                if (!ok) {
                    if (lane == 0) atomicExch(&g_tc_error, 4);
                    undone = j;
                    break;
                }
                tc_fence_after();
                // 16-column chunks of this warp's half; the next chunk's accumulators load under this one's work
                const int chunks = pad16(g.dims[l + 1]) / 16, c1 = 16 * ((half + 1) * chunks / 2);
                int c = 16 * (half * chunks / 2);
                if (c < c1) {
                    unsigned t[2][16];
                    __syncwarp();   // the TMEM loads are warp-collective
                    tmem_ld16(trow + (unsigned)c, t[0]);
                    for (; c < c1; c += 32) {
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            const int cc = c + 16 * q;
                            if (cc >= c1) break;
                            __syncwarp();
                            tmem_ld_wait(t[q]);
                            if (cc + 16 < c1) tmem_ld16(trow + (unsigned)cc + 16, t[q ^ 1]);
                            const ulonglong2* b = reinterpret_cast<const ulonglong2*>(bias + cc);
                            unsigned long long v[8];
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const ulonglong2 b4 = b[k];
                                v[2 * k] = add2(pack2(__uint_as_float(t[q][4 * k]), __uint_as_float(t[q][4 * k + 1])), b4.x);
                                v[2 * k + 1] =
                                    add2(pack2(__uint_as_float(t[q][4 * k + 2]), __uint_as_float(t[q][4 * k + 3])), b4.y);
                            }
                            if (l + 1 < g.nlayers) {
#pragma unroll
                                for (int k = 0; k < 8; ++k) v[k] = gelu2(v[k]);
                                store_group(a, r, cc, v);
                                store_group(a, r, cc + 8, v + 4);
                            } else if (row < M) {
                                store_out(g, row, cc, nout, v);
                                store_out(g, row, cc + 8, nout, v + 4);
                            }
                        }
                    }
                }
            }
        }
        if (undone < my_tiles) nan_rows(g.out, g.M, nout, undone, my_tiles, r, half);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * g.tmem_cols)
                     : "memory");
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }();
    return fn;
}

// [rows][K] BF16 row-major with leading dimension ld, boxes of box_k elements x box_rows
bool encode(CUtensorMap* map, const void* base, int K, int rows, int ld, int box_rows, int box_k = 8,
            CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_NONE) {
    auto fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dim[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t stride[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)box_k, (cuuint32_t)box_rows};
    cuuint32_t estride[2] = {1u, 1u};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dim, stride, box, estride,
              CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

std::atomic<int> g_enabled{-1};                // -1: from the environment on first use
std::atomic<unsigned long long> g_launches{0};

bool aligned16(const void* p) { return ((unsigned long long)p & 15u) == 0; }

int sm_count() {
    static const int sms = [] {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        return n < 1 ? 1 : n;
    }();
    return sms;
}

}  // namespace

bool tcgen05_gemm_enabled() {
    int e = g_enabled.load();
    if (e < 0) {
        const char* v = std::getenv("GDTK_MLP_TCGEN05");
        e = (v && std::strcmp(v, "0") == 0) ? 0 : 1;
        g_enabled.store(e);
    }
    return e != 0;
}

int tcgen05_gemm_set(int enable) {
    const int prev = tcgen05_gemm_enabled() ? 1 : 0;
    if (enable >= 0) g_enabled.store(enable ? 1 : 0);
    return prev;
}

unsigned long long tcgen05_gemm_launches() { return g_launches.load(); }

cudaError_t tcgen05_gemm_error(int* error) {
    int zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(error, g_tc_error, sizeof(int));
    if (e != cudaSuccess) return e;
    return cudaMemcpyToSymbol(g_tc_error, &zero, sizeof(int));
}

cudaError_t tcgen05_gemm_error_peek(int* error, cudaStream_t s) {
    return cudaMemcpyFromSymbolAsync(error, g_tc_error, sizeof(int), 0, cudaMemcpyDeviceToHost, s);
}

bool tcgen05_gemm_eligible(const GemmArgs& g) {
    return !g.trans_a && g.trans_b && g.alpha == 1.f && g.beta == 0.f && g.splits == 1 &&
           (g.act == ACT_NONE || g.act == ACT_GELU) && g.K % 16 == 0 && g.K >= 16 && g.K <= 256 && g.N % 16 == 0 &&
           g.N >= 16 && g.N <= 256 && g.M >= 1 && g.lda % 8 == 0 && g.ldb % 8 == 0 && g.ldd % 8 == 0 &&
           aligned16(g.A) && aligned16(g.B) && (!g.D || aligned16(g.D)) && (!g.Dh || aligned16(g.Dh)) &&
           (!g.pre || aligned16(g.pre)) && (g.D || g.Dh || g.pre);
}

// The tcgen05 form of launch_gemm_bf16 for the shapes tcgen05_gemm_eligible accepts;
// cudaErrorNotSupported when it does not apply (the caller then uses the mma.sync kernel).
cudaError_t launch_gemm_bf16_tcgen05(const GemmArgs& g, cudaStream_t s) {
    if (!tcgen05_gemm_enabled() || !tcgen05_gemm_eligible(g)) return cudaErrorNotSupported;
    alignas(64) CUtensorMap ma, mw;
    if (!encode(&ma, g.A, g.K, g.M, g.lda, TC_M) || !encode(&mw, g.B, g.K, g.N, g.ldb, g.N))
        return cudaErrorNotSupported;
    TcArgs a{};
    a.M = g.M; a.N = g.N; a.K = g.K;
    a.a_bytes = TC_M * g.K * 2;
    a.w_bytes = g.N * g.K * 2;
    unsigned cols = 32;
    while (cols < (unsigned)g.N) cols <<= 1;
    a.tmem_cols = cols;
    a.bias = g.bias; a.act = g.act; a.pre = g.pre; a.D = g.D; a.Dh = g.Dh; a.ldd = g.ldd;
    // at least 64 KB: whatever the operand sizes, every core matrix an MMA of this kernel addresses lies
    // inside the allocation
    size_t smem = (size_t)a.a_bytes + a.w_bytes + 64 + (size_t)g.N * 4;   // operands, barriers and state, bias
    if (smem < 64 * 1024) smem = 64 * 1024;
    const int sms = sm_count();
    cudaError_t e = cudaFuncSetAttribute(gemm_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int ntiles = (g.M + TC_M - 1) / TC_M;
    const int grid = ntiles < sms ? ntiles : sms;
    gemm_tc_kernel<<<grid, TC_THREADS, smem, s>>>(ma, mw, a);
    e = cudaGetLastError();
    if (e == cudaSuccess) g_launches.fetch_add(1);
    return e;
}

// The network's inference in one kernel; cudaErrorNotSupported for sizes it does not take (a layer wider than one
// accumulator's 256 columns, more layers than it has tensor maps for), which then go layer by layer.
cudaError_t launch_mlp_fused(const FusedMlp& f, cudaStream_t s) {
    if (!tcgen05_gemm_enabled() || f.nlayers < 1 || f.nlayers > FUSED_MAX_LAYERS || f.M < 1) return cudaErrorNotSupported;
    if (!aligned16(f.Xh) || !aligned16(f.X) || !aligned16(f.xs) || !aligned16(f.xd) || !aligned16(f.out) ||
        !aligned16(f.ys) || !aligned16(f.yd))
        return cudaErrorNotSupported;
    FusedMaps maps;
    FusedArgs a{};
    int kmax = 0, nmax = 0;
    for (int l = 0; l <= f.nlayers; ++l) {
        const int d = f.dims[l];
        if (d < 8 || d > 256 || d % 8) return cudaErrorNotSupported;
        a.dims[l] = d;
        if (l < f.nlayers) kmax = d > kmax ? d : kmax;
        if (l > 0) nmax = d > nmax ? d : nmax;
    }
    for (int l = 0; l < f.nlayers; ++l) {
        const int K = f.dims[l], N = f.dims[l + 1];
        if (!aligned16(f.W[l]) || !aligned16(f.bias[l]) ||
            !encode(&maps.w[l], f.W[l], K, N, K, pad16(N), FUSED_KC, CU_TENSOR_MAP_SWIZZLE_128B))
            return cudaErrorNotSupported;
        a.bias[l] = f.bias[l];
    }
    for (int l = f.nlayers; l < FUSED_MAX_LAYERS; ++l) maps.w[l] = maps.w[0];
    a.M = f.M; a.nlayers = f.nlayers;
    a.a_bytes = TC_M * pad16(kmax) * 2;
    a.stage_bytes = pad16(nmax) * FUSED_KC * 2;   // whole 1024-byte swizzle atoms: N is a multiple of 16
    unsigned cols = 32;
    while (cols < (unsigned)pad16(nmax)) cols <<= 1;
    a.tmem_cols = cols;
    const int bar_bytes = (2 * FUSED_MAX_STAGES + 8) * 8 + 2 * 256 * 4;   // barriers, biases
    a.stages = (227 * 1024 - 2 * a.a_bytes - bar_bytes) / a.stage_bytes;   // 3 of 32 KB at width 256
    if (a.stages > FUSED_MAX_STAGES) a.stages = FUSED_MAX_STAGES;
    const int smem = a.stages * a.stage_bytes + 2 * a.a_bytes + bar_bytes;
    a.Xh = f.Xh; a.X = f.X; a.xs = f.xs; a.xd = f.xd; a.out = f.out; a.ys = f.ys; a.yd = f.yd;
    a.go = f.give_up ? 0 : 1;
    cudaError_t e = cudaFuncSetAttribute(mlp_fused_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const int ntiles = (f.M - 1) / TC_M + 1, sms = sm_count();
    mlp_fused_kernel<<<ntiles < sms ? ntiles : sms, FUSED_THREADS, smem, s>>>(maps, a);
    e = cudaGetLastError();
    if (e == cudaSuccess) g_launches.fetch_add(1);
    return e;
}

}  // namespace gdtk

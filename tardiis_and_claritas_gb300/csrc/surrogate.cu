// Surrogate network of the detector signals, trained and evaluated on the GPU (no reference
// counterpart: the reference answers every scenario query with a full Monte Carlo run).
//
// Network: 6 -> 256 -> 256 -> 256 -> 256 -> 3, SiLU after each hidden layer, BF16 weights and
// activations, FP32 accumulation, FP32 master weights with Adam. In training the three 256x256 layers run
// on the 5th-generation tensor cores: one GEMM kernel computes C[M][256] = A[M][K] . B[256][K]^T with both
// operands K-major BF16, staged through shared memory in the canonical no-swizzle core-matrix layout
// and multiplied by tcgen05.mma (M=128, N=64, K=16 per instruction; a CTA makes 128 rows of 64 columns)
// into a TMEM accumulator, which the epilogue reads back with tcgen05.ld. The same kernel serves the
// forward layers (bias + SiLU epilogue), the backward-data products (SiLU-derivative epilogue) and the
// weight gradients (split-K over the batch into partial sums, which Adam adds in a fixed order). The thin
// first (6 -> 256) and last (256 -> 3) layers, the loss (added by atomics, so that its last bits depend on
// the order of the blocks), the bias gradients and the Adam update are CUDA-core kernels. Inference is one
// kernel of its own (mlp_infer_kernel) with every product on the tensor cores.
#include <cstdint>
#include <cstring>
#include <cmath>
#include <random>
#include <string>
#include <vector>
#include <algorithm>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include "claritas_gb.h"

namespace mlpk {

typedef __nv_bfloat16 bf16;

constexpr int kIn = CLR_MLP_INPUTS, kHid = CLR_MLP_WIDTH, kOut = CLR_MLP_OUTPUTS;
// flat parameter layout: W1 [256][6], b1, W2 [256][256], b2, W3, b3, W4, b4, W5 [3][256], b5
constexpr long long kOffW1 = 0, kOffB1 = kOffW1 + kHid * kIn;
constexpr long long kOffW2 = kOffB1 + kHid, kOffB2 = kOffW2 + kHid * kHid;
constexpr long long kOffW3 = kOffB2 + kHid, kOffB3 = kOffW3 + kHid * kHid;
constexpr long long kOffW4 = kOffB3 + kHid, kOffB4 = kOffW4 + kHid * kHid;
constexpr long long kOffW5 = kOffB4 + kHid, kOffB5 = kOffW5 + kOut * kHid;
constexpr long long kParams = kOffB5 + kOut;
static_assert(kParams == CLR_MLP_PARAMS, "parameter count");
// offsets of layer l's weights and biases (l = 1..5)
__host__ __device__ constexpr long long off_w(int l) {
    return l == 1 ? kOffW1 : l == 2 ? kOffW2 : l == 3 ? kOffW3 : l == 4 ? kOffW4 : kOffW5;
}
__host__ __device__ constexpr long long off_b(int l) {
    return l == 1 ? kOffB1 : l == 2 ? kOffB2 : l == 3 ? kOffB3 : l == 4 ? kOffB4 : kOffB5;
}

// ---------------- tcgen05 / mbarrier primitives (inline PTX) ----------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0u;
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Waits for the phase with the given parity to complete, for at most `limit_ns`. On time-out it
// records error code `code` and returns false (the caller cleans up and leaves).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity, int* err, int code,
                                          unsigned long long limit_ns = 2000000000ull) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    while (!mbar_try_wait(bar, parity)) {
        if (global_ns() - t0 > limit_ns) {
            if (err) atomicCAS(err, 0, code);
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// D[tmem] (+)= A[smem desc] . B[smem desc]^T, kind::f16 (BF16 inputs per the instruction descriptor)
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrive on `bar` once every tcgen05 operation this thread issued before has completed
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
// 32 lanes x 32 consecutive 32-bit columns: thread t of the warp receives lane (base lane + t)
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Shared-memory matrix descriptor of tcgen05 (no swizzle, K-major): start address, leading-dimension
// byte offset (between the two 8x16-byte core matrices along K of one instruction), stride-dimension
// byte offset (between 8-row groups), descriptor version 1 at bits 46-47, layout type 0 (no swizzle).
__host__ __device__ constexpr uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}
constexpr int kM = 128, kN = 256, kKC = 64;  // rows per tile, output width, K per shared-memory stage
// Instruction descriptor of kind::f16: D FP32 (bits 4-5 = 1), A and B BF16 (bits 7-9, 10-12 = 1), both
// K-major (bits 15, 16 = 0), N >> 3 at bits 17-22, M >> 4 at bits 24-28.
__host__ __device__ constexpr uint32_t idesc_of(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kM >> 4) << 24);
}

// The training products are small (2048 x 256 x 256), so a launch's time is a tile's own chain: operands in, MMAs,
// epilogue. A CTA takes 64 of the 256 output columns (64 CTAs for 2048 rows instead of 16), brings its whole
// K = 256 in with asynchronous copies before the first MMA (four stages of 64), and eight warps share the
// epilogue, 32 columns each. With 128 x 256 tiles, plain loads two stages deep and four warps a layer took 52 us.
// A plain product of many rows takes all 256 columns in a CTA, which then reads its rows once, in a ring of two stages
// (two CTAs share an SM with either tile). The line is where four narrow CTAs per 128 rows need a second round, two on
// each of 152 SMs (a call of K = 256 and of 1024, us, narrow / wide: 9728 rows 29.6 / 31.3 and 53.3 / 55.7, 9729 rows
// 33.2 / 32.8 and 65.1 / 56.9, 65536 rows 91.9 / 71.7 and 250.6 / 153.2).
constexpr int kGemmThreads = 256;               // warp w reads TMEM lanes 32 (w % 4) .., column half w / 4
constexpr int kStageA = kM * kKC * 2;           // 16 KB
template <int NT>                               // output columns per CTA
struct GemmTile {
    static constexpr int kStages = NT == 64 ? 4 : 2;
    static constexpr int kStageB = NT * kKC * 2;  // 8 KB, 32 KB
    static constexpr int kSmem = kStages * (kStageA + kStageB) + 64;  // stages, barriers, TMEM address
};
constexpr int kNT = 64;                         // of the training products
constexpr int kWideTiles = 2 * 152 * kNT / kN + 1;  // row tiles

enum Epi : int { EPI_STORE_F32 = 0, EPI_FWD = 1, EPI_BWD = 2 };

struct GemmArgs {
    const bf16* A;           // [M][lda], K contiguous
    long long lda;
    const bf16* B;           // [256][ldb], K contiguous
    long long ldb;
    int M, K, k_split;       // K and k_split multiples of 64; CTA y takes K columns [y*k_split, +k_split)
    const float* bias;       // [256] (EPI_FWD)
    const float* zin;        // [M][256] saved pre-activations (EPI_BWD)
    float* out_f32;          // [M][ldo]: result (STORE) or pre-activation z (FWD)
    long long ldo;
    long long part;          // STORE: CTA y's share of K goes to out_f32 + y * part
    bf16* out_bf16;          // [M][256]: silu(z) (FWD) or dz (BWD)
    bf16* out_bf16_t;        // [256][ldt]: transposed copy (FWD, BWD)
    long long ldt;
    int* err;
};
constexpr int kGemmBatch = 3;  // products of one launch (the weight gradients of the three hidden layers)
struct GemmBatch { GemmArgs g[kGemmBatch]; };

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
    const int bytes = valid ? 16 : 0;  // 0: the 16 bytes are zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
// One K chunk (64 columns) of `rows` rows into the core-matrix layout: element (r, k) at
// (r / 8) * 1024 + (k / 8) * 128 + (r % 8) * 16 + (k % 8) * 2 bytes. Rows at or past `valid` read as zero. Two
// neighbouring lanes take 32 contiguous bytes of a row, 16 lanes apart rows: whole sectors, no bank conflicts.
__device__ __forceinline__ void load_chunk(unsigned char* dst, const bf16* src, long long ld, int row0, int rows,
                                           int valid, int k0) {
    for (int q = threadIdx.x; q < rows * 8; q += kGemmThreads) {
        const int kc = (q & 1) | ((q >> 4) & 6), r = ((q >> 1) & 15) | ((q >> 7) << 4);
        const bool ok = row0 + r < valid;
        cp_async16(dst + (r >> 3) * 1024 + kc * 128 + (r & 7) * 16,
                   src + (long long)(ok ? row0 + r : 0) * ld + k0 + kc * 8, ok);
    }
}

__device__ __forceinline__ float silu_f(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float dsilu_f(float z) {
    const float s = 1.0f / (1.0f + expf(-z));
    return s * (1.0f + z * (1.0f - s));
}

template <int EPI, int NT>
__global__ void __launch_bounds__(kGemmThreads, 2) umma_gemm_kernel(GemmBatch batch) {
    constexpr int kStages = GemmTile<NT>::kStages, kStageB = GemmTile<NT>::kStageB;
    extern __shared__ __align__(1024) unsigned char sm[];
    const GemmArgs& g = batch.g[blockIdx.z / (kN / NT)];
    unsigned char* const stA0 = sm;
    unsigned char* const stB0 = sm + kStages * kStageA;
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + kStages * (kStageA + kStageB));  // [kStages]
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + kStages);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * kM, n0 = (blockIdx.z % (kN / NT)) * NT;
    const int kb = blockIdx.y * g.k_split;
    const int ke = min(g.K, kb + g.k_split);
    const int nc = ke > kb ? (ke - kb) / kKC : 0;
    auto load = [&](int c) {
        const int st = c % kStages;
        load_chunk(stA0 + st * kStageA, g.A, g.lda, m0, kM, g.M, kb + c * kKC);
        load_chunk(stB0 + st * kStageB, g.B, g.ldb, n0, NT, kN, kb + c * kKC);
    };
    for (int c = 0; c < kStages - 1; ++c) {
        if (c < nc) load(c);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (tid == 0) {
        for (int i = 0; i < kStages; ++i) mbar_init(&bar[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(tslot, NT);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    bool ok = true;
    int issued = 0;  // chunks whose MMAs were issued
    for (int c = 0; c < nc; ++c) {
        const int pc = c + kStages - 1;
        if (pc < nc) {
            // the MMAs of chunk pc - kStages read this stage: wait for their commit
            if (pc >= kStages) {
                ok = mbar_wait(&bar[pc % kStages], ((pc - kStages) / kStages) & 1, g.err, 1);
                if (!__syncthreads_and(ok)) { ok = false; break; }
            }
            load(pc);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
        fence_proxy_async();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            const uint32_t a0 = smem_u32(stA0 + (c % kStages) * kStageA), b0 = smem_u32(stB0 + (c % kStages) * kStageB);
#pragma unroll
            for (int kk = 0; kk < kKC / 16; ++kk)
                mma_bf16(tmem, smem_desc(a0 + kk * 256, 128, 1024), smem_desc(b0 + kk * 256, 128, 1024), idesc_of(NT),
                         (c > 0 || kk > 0) ? 1u : 0u);
            mma_commit(&bar[c % kStages]);
        }
        issued = c + 1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (issued > 0) {
        // the last commit covers every MMA issued before it; after a time-out wait once more (bounded)
        // so no MMA still writes the accumulator when it is released
        const bool done = mbar_wait(&bar[(issued - 1) % kStages], ((issued - 1) / kStages) & 1, g.err, 2);
        ok = ok && done;
    }
    ok = __syncthreads_and(ok);
    tc_fence_after();
    if (ok && issued > 0) {
        const int m = m0 + 32 * (warp & 3) + lane;
#pragma unroll 1
        for (int jt = (NT / 2) * (warp >> 2); jt < (NT / 2) * (warp >> 2) + NT / 2; jt += 32) {
            const int j0 = n0 + jt;
            float v[32];
            __syncwarp();
            tmem_ld32(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)jt, v);
            if (m >= g.M) continue;
            if constexpr (EPI == EPI_STORE_F32) {
                float4* o = reinterpret_cast<float4*>(g.out_f32 + blockIdx.y * g.part + (long long)m * g.ldo + j0);
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            } else if constexpr (EPI == EPI_FWD) {
                __align__(16) bf16 hb[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const float z = v[i] + g.bias[j0 + i];
                    v[i] = z;
                    hb[i] = __float2bfloat16(silu_f(z));
                }
                uint4* ho = reinterpret_cast<uint4*>(g.out_bf16 + (long long)m * kN + j0);
#pragma unroll
                for (int i = 0; i < 4; ++i) ho[i] = reinterpret_cast<const uint4*>(hb)[i];
                float4* zo = reinterpret_cast<float4*>(g.out_f32 + (long long)m * kN + j0);
#pragma unroll
                for (int i = 0; i < 8; ++i) zo[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
#pragma unroll
                for (int i = 0; i < 32; ++i) g.out_bf16_t[(long long)(j0 + i) * g.ldt + m] = hb[i];
            } else {  // EPI_BWD: dz = dh * silu'(z)
                const float4* zi = reinterpret_cast<const float4*>(g.zin + (long long)m * kN + j0);
                __align__(16) bf16 db[32];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 z = zi[i];
                    db[4 * i + 0] = __float2bfloat16(v[4 * i + 0] * dsilu_f(z.x));
                    db[4 * i + 1] = __float2bfloat16(v[4 * i + 1] * dsilu_f(z.y));
                    db[4 * i + 2] = __float2bfloat16(v[4 * i + 2] * dsilu_f(z.z));
                    db[4 * i + 3] = __float2bfloat16(v[4 * i + 3] * dsilu_f(z.w));
                }
                uint4* dout = reinterpret_cast<uint4*>(g.out_bf16 + (long long)m * kN + j0);
#pragma unroll
                for (int i = 0; i < 4; ++i) dout[i] = reinterpret_cast<const uint4*>(db)[i];
#pragma unroll
                for (int i = 0; i < 32; ++i) g.out_bf16_t[(long long)(j0 + i) * g.ldt + m] = db[i];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, NT);
    }
}

// Opt-in shared memory of every GEMM variant on the current device (called before any launch, outside
// stream capture).
static cudaError_t set_gemm_attributes() {
    const struct { const void* f; int smem; } fns[] = {
        {(const void*)umma_gemm_kernel<EPI_STORE_F32, kNT>, GemmTile<kNT>::kSmem},
        {(const void*)umma_gemm_kernel<EPI_STORE_F32, kN>, GemmTile<kN>::kSmem},
        {(const void*)umma_gemm_kernel<EPI_FWD, kNT>, GemmTile<kNT>::kSmem},
        {(const void*)umma_gemm_kernel<EPI_BWD, kNT>, GemmTile<kNT>::kSmem}};
    for (const auto& k : fns) {
        cudaError_t e = cudaFuncSetAttribute(k.f, cudaFuncAttributeMaxDynamicSharedMemorySize, k.smem);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// `count` products of one shape in one launch.
template <int EPI, int NT = kNT>
static cudaError_t launch_gemm(const GemmBatch& b, int count, int grid_y, cudaStream_t st) {
    dim3 grid((b.g[0].M + kM - 1) / kM, grid_y, count * (kN / NT));
    umma_gemm_kernel<EPI, NT><<<grid, kGemmThreads, GemmTile<NT>::kSmem, st>>>(b);
    return cudaGetLastError();
}

// ---------------- CUDA-core kernels: thin layers, loss, gradients, optimizer ----------------
__device__ __forceinline__ float bfr(float x) { return __bfloat162float(__float2bfloat16(x)); }

// Inputs of the training steps of one call, in device memory (so the captured step serves every call):
// the caller's rows and the step about to run.
struct StepArgs {
    const float *x, *t, *w;  // [rows][6], [rows][3], loss weights [rows][3] or null
    const int32_t* idx;      // row of each position, or null (position i is row i)
    int step;                // steps begun in this call; the head kernel counts it up
};
constexpr int kThinRows = 16;  // batch rows per block of the thin layers

__device__ __forceinline__ uint4 pack8(const bf16* v) { return *reinterpret_cast<const uint4*>(v); }

// Gather and layer 1 (6 -> 256): 16 rows per block, thread j one unit. Rows of z and h are stored across the
// threads, and each thread's 16 activations of its unit as two 16-byte stores of the transposed copy.
__global__ void __launch_bounds__(kHid) layer1_kernel(const StepArgs* __restrict__ a, int n, const bf16* __restrict__ w1,
                                                      const float* __restrict__ b1, float* xb, float* tb, float* wb,
                                                      float* z1, bf16* h1, bf16* h1t, long long ldt) {
    __shared__ float xs[kThinRows * kIn];
    const int r0 = blockIdx.x * kThinRows, j = threadIdx.x;
    const long long row0 = (long long)a->step * n;
    if (j < kThinRows * kIn) {
        const int r = j / kIn, i = j % kIn;
        const long long src = a->idx ? (long long)a->idx[row0 + r0 + r] : row0 + r0 + r;
        const float v = bfr(a->x[src * kIn + i]);
        xs[j] = v;
        xb[r0 * kIn + j] = v;
    } else if (j >= 128 && j < 128 + kThinRows * kOut) {
        const int q = j - 128, r = q / kOut, i = q % kOut;
        const long long src = a->idx ? (long long)a->idx[row0 + r0 + r] : row0 + r0 + r;
        tb[r0 * kOut + q] = a->t[src * kOut + i];
        wb[r0 * kOut + q] = a->w ? a->w[src * kOut + i] : 1.0f;
    }
    float w[kIn];
#pragma unroll
    for (int i = 0; i < kIn; ++i) w[i] = __bfloat162float(w1[j * kIn + i]);
    const float b = b1[j];
    __syncthreads();
    __align__(16) bf16 hv[kThinRows];
#pragma unroll
    for (int r = 0; r < kThinRows; ++r) {
        float z = b;
#pragma unroll
        for (int i = 0; i < kIn; ++i) z = fmaf(xs[r * kIn + i], w[i], z);
        hv[r] = __float2bfloat16(silu_f(z));
        h1[(long long)(r0 + r) * kHid + j] = hv[r];
        z1[(long long)(r0 + r) * kHid + j] = z;
    }
    uint4* o = reinterpret_cast<uint4*>(h1t + (long long)j * ldt + r0);
    o[0] = pack8(hv);
    o[1] = pack8(hv + 8);
}

// Output layer (256 -> 3), one warp per row (16 rows per block): the loss L = sum w (y - t)^2 / (3 n), dy = dL/dy
// and the gradient through the output layer into the last hidden layer (dz4 = (dy . W5) * silu'(z4)); the
// transposed copy goes through shared memory, the loss is added once per block.
__global__ void __launch_bounds__(256) head_kernel(StepArgs* a, const bf16* __restrict__ h4, const float* __restrict__ z4,
                                                   int n, const bf16* __restrict__ w5, const float* __restrict__ b5,
                                                   const float* __restrict__ tb, const float* __restrict__ wb, float* dy,
                                                   bf16* dz4, bf16* dz4t, long long ldt, float* loss_sum) {
    __shared__ __align__(16) bf16 tile[kThinRows][kHid + 8];  // stored 16 bytes at a time
    __shared__ float block_loss[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r0 = blockIdx.x * kThinRows;
    if (blockIdx.x == 0 && threadIdx.x == 0) a->step += 1;
    float wv[kOut][8], lsum = 0.0f;
#pragma unroll
    for (int k = 0; k < kOut; ++k)
#pragma unroll
        for (int i = 0; i < 8; ++i) wv[k][i] = __bfloat162float(w5[k * kHid + lane * 8 + i]);
    const float scale = 2.0f / (3.0f * (float)n);
#pragma unroll
    for (int q = 0; q < kThinRows / 8; ++q) {
        const int lr = warp + 8 * q, r = r0 + lr;
        float hv[8], acc[kOut] = {0.0f, 0.0f, 0.0f};
        const uint4 hq = *reinterpret_cast<const uint4*>(h4 + (long long)r * kHid + lane * 8);
        const float4 za = *reinterpret_cast<const float4*>(z4 + (long long)r * kHid + lane * 8),
                     zb = *reinterpret_cast<const float4*>(z4 + (long long)r * kHid + lane * 8 + 4);
        const float zv[8] = {za.x, za.y, za.z, za.w, zb.x, zb.y, zb.z, zb.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) hv[i] = __bfloat162float(reinterpret_cast<const bf16*>(&hq)[i]);
#pragma unroll
        for (int k = 0; k < kOut; ++k) {
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[k] = fmaf(hv[i], wv[k][i], acc[k]);
            for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
        }
        float d[kOut], l = 0.0f;
#pragma unroll
        for (int k = 0; k < kOut; ++k) {
            const float e = acc[k] + b5[k] - tb[r * kOut + k];
            const float we = wb[r * kOut + k] * e;
            d[k] = scale * we;
            l += we * e;
        }
        lsum += l;
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < kOut; ++k) dy[r * kOut + k] = d[k];
        }
        __align__(16) bf16 dv[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float g = 0.0f;
#pragma unroll
            for (int k = 0; k < kOut; ++k) g = fmaf(d[k], wv[k][i], g);
            dv[i] = __float2bfloat16(g * dsilu_f(zv[i]));
        }
        *reinterpret_cast<uint4*>(dz4 + (long long)r * kHid + lane * 8) = pack8(dv);
        *reinterpret_cast<uint4*>(&tile[lr][lane * 8]) = pack8(dv);
    }
    if (lane == 0) block_loss[warp] = lsum;
    __syncthreads();
    __align__(16) bf16 col[kThinRows];
#pragma unroll
    for (int r = 0; r < kThinRows; ++r) col[r] = tile[r][threadIdx.x];
    uint4* o = reinterpret_cast<uint4*>(dz4t + (long long)threadIdx.x * ldt + r0);
    o[0] = pack8(col);
    o[1] = pack8(col + 8);
    if (threadIdx.x == 0) {
        float l = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; ++w) l += block_loss[w];
        atomicAdd(loss_sum, l);
    }
}

// Small gradient reductions over the batch, a thread per unit and 256 rows, each row after the other; a unit's rows
// are contiguous in the transposed copies and come in 16 bytes at a time, 64 rows ahead; the rows' inputs and
// output gradients are staged in shared memory (a thread that loads them row by row waits for memory at each):
//   db_l[j] = sum_r dz_l[r][j] (l = 1..4), with it for l = 1 dW1[j][i] = sum_r dz1[r][j] x[r][i];
//   dW5[k][j] = sum_r dy[r][k] h4[r][j]; and one thread for db5[k] = sum_r dy[r][k].
// A block's sums go to its own row of partial sums (`parts`); they are added in the rows' order where the gradient is
// used, so a step does not depend on which block ends first (added with atomics, two runs of an epoch differed by up
// to 5e-5 of the largest weight, Adam's first steps being the signs of the gradients).
constexpr int kHiddenW = 3 * kHid * kHid, kSmallParams = (int)kParams - kHiddenW;
constexpr int kWeightRows = 512;  // batch rows of a partial sum of W2..W4
struct GradParts {
    const float* hidden;  // [n_hidden][3][256][256]: W2, W3, W4
    const float* rest;    // [n_rest][kSmallParams]: the other parameters in their order
    int n_hidden, n_rest;
};
__host__ __device__ constexpr int rest_index(int p) {
    return p - kHid * kHid * ((p >= (int)off_b(2)) + (p >= (int)off_b(3)) + (p >= (int)off_b(4)));
}
static_assert(rest_index((int)kParams - 1) == kSmallParams - 1, "the parameters outside W2..W4, gap-free");
__device__ __forceinline__ float grad_of(const GradParts& G, int p) {
    const float* src = G.rest + rest_index(p);
    int rows = G.n_rest;
    long long stride = kSmallParams;
#pragma unroll
    for (int l = 2; l <= 4; ++l)
        if (p >= (int)off_w(l) && p < (int)off_b(l)) {
            src = G.hidden + (l - 2) * kHid * kHid + (p - (int)off_w(l));
            rows = G.n_hidden;
            stride = kHiddenW;
        }
    float g = 0.0f;
#pragma unroll 4
    for (int i = 0; i < rows; ++i) g += src[i * stride];
    return g;
}
__global__ void sum_grads_kernel(GradParts G, float* grads) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < (int)kParams) grads[p] = grad_of(G, p);
}
constexpr int kSmallUnits = 5 * kHid + 1;
constexpr int kSmallRows = 256;
constexpr int kSmallThreads = 64;
__global__ void __launch_bounds__(kSmallThreads) small_grads_kernel(const bf16* const* __restrict__ dzt,
                                                                    const bf16* __restrict__ h4t, long long ldt,
                                                                    const float* __restrict__ xb,
                                                                    const float* __restrict__ dy, int n, float* parts) {
    __shared__ float xs[kSmallRows * kIn], ds[kSmallRows * kOut];
    const int r0 = blockIdx.y * kSmallRows, rows = min(n - r0, kSmallRows);  // a multiple of 128
    const int unit = blockIdx.x * kSmallThreads + threadIdx.x;
    const int what = unit / kHid, j = unit % kHid;  // 0..3: layer what + 1; 4: output weights; 5: output bias
    if (what == 0)
        for (int i = threadIdx.x; i < rows * kIn; i += kSmallThreads) xs[i] = xb[r0 * kIn + i];
    if (what >= 4)
        for (int i = threadIdx.x; i < rows * kOut; i += kSmallThreads) ds[i] = dy[r0 * kOut + i];
    __syncthreads();
    if (unit >= kSmallUnits) return;
    const uint4* row = reinterpret_cast<const uint4*>((what < 4 ? dzt[what] : h4t) + (long long)j * ldt + r0);
    float s[1 + kIn] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    if (what == 5) {
#pragma unroll 8
        for (int r = 0; r < rows; ++r)
#pragma unroll
            for (int k = 0; k < kOut; ++k) s[k] += ds[r * kOut + k];
    } else {
        for (int r = 0; r < rows; r += 64) {
            uint4 q[8];
#pragma unroll
            for (int h = 0; h < 8; ++h) q[h] = row[r / 8 + h];
#pragma unroll
            for (int h = 0; h < 64; ++h) {
                const float v = __bfloat162float(reinterpret_cast<const bf16*>(q)[h]);
                if (what == 4) {
#pragma unroll
                    for (int k = 0; k < kOut; ++k) s[k] = fmaf(ds[(r + h) * kOut + k], v, s[k]);
                } else {
                    s[kIn] += v;
                    if (what == 0) {
#pragma unroll
                        for (int i = 0; i < kIn; ++i) s[i] = fmaf(v, xs[(r + h) * kIn + i], s[i]);
                    }
                }
            }
        }
    }
    float* const out = parts + (long long)blockIdx.y * kSmallParams;
    if (what < 4) {
        out[rest_index((int)off_b(what + 1) + j)] = s[kIn];
        if (what == 0)
#pragma unroll
            for (int i = 0; i < kIn; ++i) out[rest_index((int)kOffW1 + j * kIn + i)] = s[i];
    } else {
#pragma unroll
        for (int k = 0; k < kOut; ++k) out[rest_index((int)(what == 4 ? kOffW5 + k * kHid + j : kOffB5 + k))] = s[k];
    }
}

// BF16 copies of the weights: w[l] = W_l as [out][in] and wt[l] = W_l^T as [in][out] (l = 2..4), plus
// W1 and W5 as [out][in]. One thread per parameter.
struct PackArgs {
    bf16* w[6];
    bf16* wt[6];
    bf16* wp[6];  // l = 2..4: the shared-memory image of W_l as a B operand (256 x 256 core-matrix layout)
};
// element (r, k) of a K = 256 operand image in the core-matrix layout (8 x 16-byte core matrices, K-adjacent
// core matrices 128 bytes apart, 8-row groups 4096 bytes apart), in BF16 elements
__host__ __device__ __forceinline__ int img_idx(int r, int k) {
    return ((r >> 3) * 4096 + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2) >> 1;
}
__device__ __forceinline__ void pack_one(const PackArgs& pa, int p, float v) {
    const bf16 b = __float2bfloat16(v);
    if (p < (int)kOffB1) {
        const int out = p / kIn, in = p % kIn;
        pa.w[1][p] = b;
        // 256 x 16 image (K = 16): 8-row groups 256 bytes apart
        pa.wp[1][((out >> 3) * 256 + (in >> 3) * 128 + (out & 7) * 16 + (in & 7) * 2) >> 1] = b;
    } else if (p < (int)kOffW5) {
        // layers 2..4: weights and biases repeat every 256 x 256 + 256 parameters
        constexpr int kStep = (int)(kOffW3 - kOffW2);
        const int l = 2 + (p - (int)kOffW2) / kStep, o = (p - (int)kOffW2) % kStep;
        if (p < (int)kOffW2 || o >= kHid * kHid) return;  // a bias
        const int out = o / kHid, in = o % kHid;
        pa.w[l][o] = b;
        pa.wt[l][in * kHid + out] = b;
        pa.wp[l][img_idx(out, in)] = b;
    } else if (p < (int)kOffB5) {
        const int o = p - (int)kOffW5;
        pa.w[5][o] = b;
        pa.wp[5][img_idx(o / kHid, o % kHid)] = b;  // 16 x 256, rows 3..15 stay zero
    }
}
static_assert(kOffW4 - kOffW3 == kOffW3 - kOffW2 && kOffW5 - kOffW4 == kOffW3 - kOffW2, "hidden layers are equally spaced");
__global__ void pack_kernel(const float* __restrict__ params, PackArgs pa) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < (int)kParams) pack_one(pa, p, params[p]);
}

// Adam (bias-corrected) on every parameter, whose gradient it adds up from the step's partial sums; then the BF16
// copies are refreshed. hp: per step of the call the learning rate and the two bias corrections.
__global__ void adam_kernel(float* params, GradParts G, float* m1, float* m2, const StepArgs* __restrict__ step,
                            const float4* __restrict__ hp, PackArgs pa) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (int)kParams) return;
    const float4 h = hp[step->step - 1];
    const float lr = h.x, c1 = h.y, c2 = h.z;
    const float g = grad_of(G, p);
    const float a = 0.9f * m1[p] + 0.1f * g;
    const float b = 0.999f * m2[p] + 0.001f * g * g;
    m1[p] = a;
    m2[p] = b;
    const float v = params[p] - lr * (a / c1) / (sqrtf(b / c2) + 1e-8f);
    params[p] = v;
    pack_one(pa, p, v);
}

// ---------------- fused inference: every layer of a 128-row tile on one SM ----------------
// A persistent CTA per SM walks 128-row tiles with every product on the tensor cores: layer 1 with K padded from 6
// to 16, three 256x256 layers, the 256 -> 3 output layer with N padded to 16. What bounds it is the SiLU: one
// multi-function operation per activation, 16 a clock and SM, 2048 cycles per layer and tile, against 1024 for the
// layer's MMAs. So the MMAs run under the epilogues: a layer's 256 outputs are two halves of 128 columns; while
// sixteen warps turn half 0 of layer l into activations, a warp of its own has the tensor cores make half 1, and
// while they work on half 1, the first half of layer l + 1's K. Activations stay in tensor memory (two images of
// 128 columns, the accumulator the other 256), from where tcgen05.mma takes its A operand, which leaves shared
// memory to the weights: a ring of three half layers (64 KB each, one bulk copy), refilled as each half's MMAs end.
// With the activations in shared memory, one weight buffer and each layer's MMAs, copy and epilogue one after the
// other, 65536 queries took 52 us; now 40.4 us (a call 80.8 -> 74.1 us). What is left is the chain half of MMAs ->
// half epilogue of a tile, about 10 us, of which 131072 tanh on the multi-function unit take 4.3.
constexpr int kInferWarps = 16;                  // epilogue warps: TMEM lane quarter w % 4, 32 columns of each half
constexpr int kInferThreads = 32 * (kInferWarps + 1);  // and one warp that issues copies and MMAs
constexpr int kHalf = kHid / 2;
constexpr int kWHalfBytes = kHalf * kHid * 2;    // 64 KB: rows of one half of a 256x256 weight image
constexpr int kWSlots = 3;
constexpr int kXBytes = kM * 16 * 2;             // 4 KB: the tile's inputs, K padded to 16
constexpr int kW1Bytes = kHid * 16 * 2;          // 8 KB: W1 image, 256 x 16
constexpr int kW5Bytes = 16 * kHid * 2;          // 8 KB: W5 image, 16 (3 used) x 256
constexpr int kOffSmX = kWSlots * kWHalfBytes;
constexpr int kOffSmW1 = kOffSmX + kXBytes;
constexpr int kOffSmW5 = kOffSmW1 + kW1Bytes;
constexpr int kOffSmBias = kOffSmW5 + kW5Bytes;              // f32 [4][256]: b1..b4
constexpr int kOffSmB5 = kOffSmBias + 4 * kHid * 4;          // f32 [4]
constexpr int kOffSmBar = kOffSmB5 + 16;
constexpr int kInferBars = kWSlots + 2 + 2 + 3;  // weights arrived; half done; activations written; inputs, output, end
constexpr int kOffSmSlot = kOffSmBar + 8 * kInferBars;       // TMEM address
constexpr int kInferSmem = kOffSmSlot + 16;
static_assert(kOffSmBar % 8 == 0 && kInferSmem <= 227 * 1024, "shared-memory plan");
// tensor memory: two activation images (BF16 pairs, K = 256 in 128 columns), the accumulator
constexpr uint32_t kTmemD = 2 * kHalf, kTmemCols = 512;

struct InferArgs {
    const float* x;      // [n][6]
    float* y;            // [n][3]
    long long n;
    int tiles;
    const bf16* wp[3];   // images of W2, W3, W4 (256 x 256; half h is its rows 128 h .., contiguous)
    const bf16* w1p;     // image of W1 padded to 256 x 16
    const bf16* w5p;     // image of W5 padded to 16 x 256
    const float* params;
    int* err;
};

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// silu(z) = z/2 (1 + tanh(z/2)): one multi-function-unit operation per element (hardware tanh approximation,
// relative error far below the BF16 rounding that follows)
__device__ __forceinline__ float silu_tanh(float z) {
    const float h = 0.5f * z;
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(h));
    return fmaf(h, t, h);
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float* v) {
    uint32_t r0, r1, r2, r3;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    v[0] = __uint_as_float(r0); v[1] = __uint_as_float(r1); v[2] = __uint_as_float(r2); v[3] = __uint_as_float(r3);
}

// D[tmem] (+)= A[tmem] . B[smem desc]^T: the A operand from tensor memory (lane = row, two BF16 of K per column)
__device__ __forceinline__ void mma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__global__ void __launch_bounds__(kInferThreads, 1) mlp_infer_kernel(InferArgs a) {
    extern __shared__ __align__(1024) unsigned char sm[];
    unsigned char* X = sm + kOffSmX;
    float* bs = reinterpret_cast<float*>(sm + kOffSmBias);
    float* b5s = reinterpret_cast<float*>(sm + kOffSmB5);
    uint64_t* const wfull = reinterpret_cast<uint64_t*>(sm + kOffSmBar);  // [3] a weight half arrived in its slot
    uint64_t* const dfull = wfull + kWSlots;                              // [2] the MMAs of a half of D completed
    uint64_t* const aready = dfull + 2;  // [2] a half of D was read and its activations written (per epilogue warp)
    uint64_t* const xready = aready + 2;  // the tile's inputs are in X and the previous output was read
    uint64_t* const yfull = xready + 1;   // the output layer's MMAs completed
    uint64_t* const drained = yfull + 1;  // every MMA issued has completed
    uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + kOffSmSlot);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    {
        const uint4* s1 = reinterpret_cast<const uint4*>(a.w1p);
        const uint4* s5 = reinterpret_cast<const uint4*>(a.w5p);
        uint4* d1 = reinterpret_cast<uint4*>(sm + kOffSmW1);
        uint4* d5 = reinterpret_cast<uint4*>(sm + kOffSmW5);
        for (int i = tid; i < kW1Bytes / 16; i += kInferThreads) d1[i] = s1[i];
        for (int i = tid; i < kW5Bytes / 16; i += kInferThreads) d5[i] = s5[i];
    }
    for (int i = tid; i < 4 * kHid; i += kInferThreads) bs[i] = a.params[off_b(1 + i / kHid) + i % kHid];
    if (tid < kOut) b5s[tid] = a.params[kOffB5 + tid];
    if (tid == 0) {
        for (int i = 0; i < kWSlots; ++i) mbar_init(&wfull[i], 1);
        for (int h = 0; h < 2; ++h) {
            mbar_init(&dfull[h], 1);
            mbar_init(&aready[h], kInferWarps);
        }
        mbar_init(xready, 4);  // the four warps that hold column group 0
        mbar_init(yfull, 1);
        mbar_init(drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(tslot, kTmemCols);
    fence_proxy_async();  // the weight images written above
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    const int my_tiles = (int)blockIdx.x < a.tiles ? (a.tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    if (warp == kInferWarps) {
        // ---- copies and MMAs (one thread) ----
        if (lane == 0) {
            const uint32_t sW = smem_u32(sm), sX = smem_u32(X);
            const uint32_t sW1 = smem_u32(sm + kOffSmW1), sW5 = smem_u32(sm + kOffSmW5);
            const int halves = 6 * my_tiles;  // weight halves in the order they are used
            int loaded = 0, used = 0;
            auto refill = [&]() {
                if (loaded >= halves) return;
                const int i = loaded % 6, slot = loaded % kWSlots;
                bulk_load(sm + slot * kWHalfBytes, a.wp[i >> 1] + (size_t)(i & 1) * kHalf * kHid, kWHalfBytes, &wfull[slot]);
                ++loaded;
            };
            for (int i = 0; i < kWSlots; ++i) refill();
            unsigned dphase = 0, aphase = 0;  // completed phases of dfull (both halves alike) and of aready
            bool ok = true;
            for (int t = 0; t < my_tiles && ok; ++t) {
                if (!(ok = mbar_wait(xready, t & 1, a.err, 4))) break;
                tc_fence_after();
                for (int h = 0; h < 2; ++h) {  // layer 1: K = 16, inputs from shared memory
                    mma_bf16(tmem + kTmemD + h * kHalf, smem_desc(sX, 128, 256), smem_desc(sW1 + h * 4096, 128, 256),
                             idesc_of(kHalf), 0u);
                    mma_commit(&dfull[h]);
                }
                ++dphase;
                for (int l = 0; l < 3 && ok; ++l) {
                    const uint32_t act = tmem + (l & 1) * kHalf;  // activations of the previous layer
                    for (int h = 0; h < 2 && ok; ++h) {
                        const int slot = used % kWSlots;
                        if (!(ok = mbar_wait(&wfull[slot], (used / kWSlots) & 1, a.err, 3))) break;
                        const uint32_t w = sW + slot * kWHalfBytes, d = tmem + kTmemD + h * kHalf;
                        for (int kh = 0; kh < 2 && ok; ++kh) {
                            // K half kh needs activation half kh; the accumulator half h was read when both are there
                            if (h == 0) {
                                if (!(ok = mbar_wait(&aready[kh], aphase & 1, a.err, 5))) break;
                                tc_fence_after();
                            }
#pragma unroll
                            for (int kk = 8 * kh; kk < 8 * kh + 8; ++kk)
                                mma_bf16_ts(d, act + kk * 8, smem_desc(w + kk * 256, 128, 4096), idesc_of(kHalf),
                                            kk > 0 ? 1u : 0u);
                        }
                        if (ok) mma_commit(&dfull[h]);
                        ++used;
                    }
                    if (!ok) break;
                    ++aphase;
                    for (int h = 0; h < 2 && ok; ++h) {  // a half's MMAs completed: its slot takes the next half in line
                        ok = mbar_wait(&dfull[h], dphase & 1, a.err, 6);
                        if (ok) refill();
                    }
                    ++dphase;
                }
                if (!ok) break;
                for (int kh = 0; kh < 2 && ok; ++kh) ok = mbar_wait(&aready[kh], aphase & 1, a.err, 5);
                if (!ok) break;
                ++aphase;
                tc_fence_after();
#pragma unroll
                for (int kk = 0; kk < kHid / 16; ++kk)
                    mma_bf16_ts(tmem + kTmemD, tmem + kHalf + kk * 8, smem_desc(sW5 + kk * 256, 128, 4096), idesc_of(16),
                                kk > 0 ? 1u : 0u);
                mma_commit(yfull);
            }
            // MMAs and (only after a failed wait) weight copies in flight must end before the CTA leaves
            mma_commit(drained);
            (void)mbar_wait(drained, 0, a.err, 10);
            for (; used < loaded; ++used) (void)mbar_wait(&wfull[used % kWSlots], (used / kWSlots) & 1, a.err, 7);
        }
    } else {
        // ---- inputs, epilogues, outputs ----
        const int quarter = warp & 3, cgroup = warp >> 2;
        const int r = quarter * 32 + lane;  // this thread's row of the tile (and TMEM lane)
        const uint32_t tlane = tmem + ((uint32_t)(quarter * 32) << 16);
        float xv[kIn];
        auto fetch = [&](int t) {  // the inputs of this CTA's tile t
            const long long row = ((long long)blockIdx.x + (long long)t * gridDim.x) * kM + r;
#pragma unroll
            for (int i = 0; i < kIn; ++i) xv[i] = t < my_tiles && row < a.n ? a.x[row * kIn + i] : 0.0f;
        };
        auto put = [&]() {  // a 128 x 16 A image (K 6..15 zero)
            uint4 lo;
            lo.x = pack_bf16x2(xv[0], xv[1]);
            lo.y = pack_bf16x2(xv[2], xv[3]);
            lo.z = pack_bf16x2(xv[4], xv[5]);
            lo.w = 0u;
            *reinterpret_cast<uint4*>(X + (r >> 3) * 256 + (r & 7) * 16) = lo;
            *reinterpret_cast<uint4*>(X + (r >> 3) * 256 + 128 + (r & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
            fence_proxy_async();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(xready);
        };
        if (cgroup == 0 && my_tiles > 0) {
            fetch(0);
            put();
        }
        bool ok = true;
        unsigned dphase = 0;
        for (int t = 0; t < my_tiles && ok; ++t) {
            if (cgroup == 0) fetch(t + 1);
            for (int l = 0; l < 4 && ok; ++l) {  // epilogue of hidden layer l + 1 into activation image l & 1
                for (int h = 0; h < 2; ++h) {
                    if (!(ok = __all_sync(0xffffffffu, mbar_wait(&dfull[h], dphase & 1, a.err, 8)))) break;
                    tc_fence_after();
                    const int j0 = h * kHalf + cgroup * 32;
                    const float* bias = bs + l * kHid + j0;
                    float v[32];
                    tmem_ld32(tlane + kTmemD + (uint32_t)j0, v);
                    uint32_t o[16];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const float4 b = *reinterpret_cast<const float4*>(bias + 4 * q);
                        o[2 * q] = pack_bf16x2(silu_tanh(v[4 * q] + b.x), silu_tanh(v[4 * q + 1] + b.y));
                        o[2 * q + 1] = pack_bf16x2(silu_tanh(v[4 * q + 2] + b.z), silu_tanh(v[4 * q + 3] + b.w));
                    }
                    tmem_st16(tlane + (uint32_t)((l & 1) * kHalf + j0 / 2), o);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&aready[h]);
                }
                ++dphase;
            }
            if (!ok) break;
            if (cgroup == 0) {
                if (!(ok = __all_sync(0xffffffffu, mbar_wait(yfull, t & 1, a.err, 9)))) break;
                tc_fence_after();
                float v[4];
                tmem_ld4(tlane + kTmemD, v);
                const long long row = ((long long)blockIdx.x + (long long)t * gridDim.x) * kM + r;
                if (row < a.n)
#pragma unroll
                    for (int k = 0; k < kOut; ++k) a.y[row * kOut + k] = v[k] + b5s[k];
                if (t + 1 < my_tiles) put();
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

}  // namespace mlpk

using namespace mlpk;

// ---------------- the network object behind the C ABI ----------------
struct clr_mlp {
    int device = 0, num_sms = 0;
    cudaStream_t stream = nullptr;
    int cap = 0;  // batch rows of the work buffers (multiple of 128)
    std::string err;
    std::vector<void*> allocs;
    float *params = nullptr, *grads = nullptr, *m1 = nullptr, *m2 = nullptr;
    float *hidden_parts = nullptr, *rest_parts = nullptr;  // partial gradients of a step (GradParts)
    PackArgs pa{};
    float* z[5] = {};          // [cap][256] pre-activations of hidden layers 1..4
    bf16* h[5] = {};           // [cap][256] activations
    bf16* ht[5] = {};          // [256][cap] transposed activations
    bf16* dz[5] = {};          // [cap][256] gradients at the pre-activations
    bf16* dzt[5] = {};         // [256][cap]
    const bf16** d_dzt = nullptr;  // device array of dzt[1..4]
    float *xb = nullptr, *tb = nullptr, *dy = nullptr, *loss = nullptr;
    float* wb = nullptr;          // [cap][3] loss weights of the batch rows
    const float* d_w = nullptr;   // the caller's loss weights (clr_mlp_set_loss_weights), or null
    int* d_err = nullptr;
    long long steps = 0;
    float last_ms = 0.0f;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaStream_t side = nullptr;  // the small gradient reductions
    cudaEvent_t fork = nullptr, join = nullptr;
    // the captured training step of batch size step_n; its inputs are read from device memory
    cudaGraphExec_t step_exec = nullptr;
    int step_n = 0;
    StepArgs* d_step = nullptr;
    float4* d_hp = nullptr;  // lr, c1, c2 of every step of the call
    long long hp_cap = 0;
};

static int mfail(clr_mlp* m, int code, const char* msg) {
    if (m) m->err = msg;
    return code;
}
#define MCU(call)                                                                           \
    do {                                                                                    \
        cudaError_t e_ = (call);                                                            \
        if (e_ != cudaSuccess) {                                                            \
            if (m) m->err = std::string(#call) + ": " + cudaGetErrorString(e_);             \
            return CLR_ERR_CUDA;                                                            \
        }                                                                                   \
    } while (0)

static cudaError_t malloc_tracked(clr_mlp* m, void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaSuccess) m->allocs.push_back(*p);
    return e;
}

// Forward pass of the n rows (a multiple of 128, n <= cap) that d_step names; pre-activations and transposed
// activations are kept for the backward pass.
static cudaError_t forward_rows(clr_mlp* m, int n, cudaStream_t st) {
    layer1_kernel<<<n / kThinRows, kHid, 0, st>>>(m->d_step, n, m->pa.w[1], m->params + kOffB1, m->xb, m->tb, m->wb,
                                                  m->z[1], m->h[1], m->ht[1], m->cap);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    for (int l = 2; l <= 4; ++l) {
        GemmBatch b{};
        GemmArgs& g = b.g[0];
        g.A = m->h[l - 1]; g.lda = kHid; g.B = m->pa.w[l]; g.ldb = kHid;
        g.M = n; g.K = kHid; g.k_split = kHid;
        g.bias = m->params + off_b(l);
        g.out_f32 = m->z[l]; g.ldo = kHid; g.out_bf16 = m->h[l]; g.out_bf16_t = m->ht[l]; g.ldt = m->cap;
        g.err = m->d_err;
        if ((e = launch_gemm<EPI_FWD>(b, 1, 1, st)) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Backward pass of the n rows of the last forward (targets in tb): gradients as partial sums (grad_parts).
static cudaError_t backward_rows(clr_mlp* m, int n, cudaStream_t st) {
    head_kernel<<<n / kThinRows, 256, 0, st>>>(m->d_step, m->h[4], m->z[4], n, m->pa.w[5], m->params + kOffB5, m->tb,
                                               m->wb, m->dy, m->dz[4], m->dzt[4], m->cap, m->loss);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    for (int l = 4; l >= 2; --l) {  // dz_{l-1} = (dz_l . W_l) * silu'(z_{l-1})
        GemmBatch b{};
        GemmArgs& g = b.g[0];
        g.A = m->dz[l]; g.lda = kHid; g.B = m->pa.wt[l]; g.ldb = kHid;
        g.M = n; g.K = kHid; g.k_split = kHid;
        g.zin = m->z[l - 1]; g.out_bf16 = m->dz[l - 1]; g.out_bf16_t = m->dzt[l - 1]; g.ldt = m->cap;
        g.err = m->d_err;
        if ((e = launch_gemm<EPI_BWD>(b, 1, 1, st)) != cudaSuccess) return e;
    }
    // the small reductions run beside the weight gradients
    if ((e = cudaEventRecord(m->fork, st)) != cudaSuccess) return e;
    if ((e = cudaStreamWaitEvent(m->side, m->fork, 0)) != cudaSuccess) return e;
    small_grads_kernel<<<dim3((kSmallUnits + kSmallThreads - 1) / kSmallThreads, (n + kSmallRows - 1) / kSmallRows),
                         kSmallThreads, 0, m->side>>>(m->d_dzt, m->ht[4], m->cap, m->xb, m->dy, n, m->rest_parts);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = cudaEventRecord(m->join, m->side)) != cudaSuccess) return e;
    GemmBatch b{};
    for (int l = 2; l <= 4; ++l) {  // dW_l = dz_l^T . h_{l-1}, split over the batch, the three layers in one launch
        GemmArgs& g = b.g[l - 2];
        g.A = m->dzt[l]; g.lda = m->cap; g.B = m->ht[l - 1]; g.ldb = m->cap;
        g.M = kHid; g.K = n; g.k_split = kWeightRows;
        g.out_f32 = m->hidden_parts + (l - 2) * kHid * kHid; g.ldo = kHid; g.part = kHiddenW; g.err = m->d_err;
    }
    if ((e = launch_gemm<EPI_STORE_F32>(b, kGemmBatch, (n + kWeightRows - 1) / kWeightRows, st)) != cudaSuccess) return e;
    return cudaStreamWaitEvent(st, m->join, 0);
}

static GradParts grad_parts(const clr_mlp* m, int n) {
    return {m->hidden_parts, m->rest_parts, (n + kWeightRows - 1) / kWeightRows, (n + kSmallRows - 1) / kSmallRows};
}

static int check_dev(clr_mlp* m) {
    int herr = 0;
    MCU(cudaMemcpyAsync(&herr, m->d_err, sizeof(int), cudaMemcpyDeviceToHost, m->stream));
    MCU(cudaStreamSynchronize(m->stream));
    if (herr) {
        MCU(cudaMemsetAsync(m->d_err, 0, sizeof(int), m->stream));
        return mfail(m, CLR_ERR_DEVICE_TIMEOUT, "tensor-core GEMM timed out waiting for its MMAs");
    }
    return CLR_OK;
}

extern "C" {

int clr_mlp_create(clr_mlp** out, int device, int max_batch, uint64_t seed) {
    if (!out || max_batch < 128 || max_batch % 128) return CLR_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    clr_mlp* m = new clr_mlp();
    m->device = device;
    m->cap = max_batch;
    MCU(cudaSetDevice(device));
    MCU(cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking));
    MCU(set_gemm_attributes());
    MCU(cudaFuncSetAttribute(mlp_infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kInferSmem));
    MCU(cudaDeviceGetAttribute(&m->num_sms, cudaDevAttrMultiProcessorCount, device));
    MCU(cudaEventCreate(&m->ev0));
    MCU(cudaEventCreate(&m->ev1));
    MCU(cudaStreamCreateWithFlags(&m->side, cudaStreamNonBlocking));
    MCU(cudaEventCreateWithFlags(&m->fork, cudaEventDisableTiming));
    MCU(cudaEventCreateWithFlags(&m->join, cudaEventDisableTiming));
    auto F = [&](float** p, size_t cnt) { return malloc_tracked(m, (void**)p, cnt * sizeof(float)); };
    auto H = [&](bf16** p, size_t cnt) { return malloc_tracked(m, (void**)p, cnt * sizeof(bf16)); };
    MCU(F(&m->params, kParams)); MCU(F(&m->grads, kParams)); MCU(F(&m->m1, kParams)); MCU(F(&m->m2, kParams));
    for (int l = 1; l <= 5; ++l) {
        const int nin = l == 1 ? kIn : kHid, nout = l == 5 ? kOut : kHid;
        MCU(H(&m->pa.w[l], (size_t)nin * nout));
        if (l >= 2 && l <= 4) {
            MCU(H(&m->pa.wt[l], (size_t)nin * nout));
            MCU(H(&m->pa.wp[l], (size_t)nin * nout));
        }
        if (l == 1 || l == 5) {  // padded images: zero padding written once, weights by every pack
            MCU(H(&m->pa.wp[l], (size_t)kHid * 16));
            MCU(cudaMemset(m->pa.wp[l], 0, (size_t)kHid * 16 * sizeof(bf16)));
        }
    }
    const GradParts most = grad_parts(m, m->cap);
    MCU(F(&m->hidden_parts, (size_t)most.n_hidden * kHiddenW));
    MCU(F(&m->rest_parts, (size_t)most.n_rest * kSmallParams));
    const size_t act = (size_t)m->cap * kHid;
    for (int l = 1; l <= 4; ++l) {
        MCU(F(&m->z[l], act)); MCU(H(&m->h[l], act)); MCU(H(&m->ht[l], act));
        MCU(H(&m->dz[l], act)); MCU(H(&m->dzt[l], act));
    }
    MCU(F(&m->xb, (size_t)m->cap * kIn)); MCU(F(&m->tb, (size_t)m->cap * kOut)); MCU(F(&m->wb, (size_t)m->cap * kOut));
    MCU(F(&m->dy, (size_t)m->cap * kOut)); MCU(F(&m->loss, 4));
    MCU(malloc_tracked(m, (void**)&m->d_err, sizeof(int)));
    MCU(malloc_tracked(m, (void**)&m->d_dzt, 4 * sizeof(bf16*)));
    MCU(malloc_tracked(m, (void**)&m->d_step, sizeof(StepArgs)));
    const bf16* dzt[4] = {m->dzt[1], m->dzt[2], m->dzt[3], m->dzt[4]};
    MCU(cudaMemcpy(m->d_dzt, dzt, sizeof dzt, cudaMemcpyHostToDevice));
    MCU(cudaMemset(m->d_err, 0, sizeof(int)));
    MCU(cudaMemset(m->m1, 0, kParams * sizeof(float)));
    MCU(cudaMemset(m->m2, 0, kParams * sizeof(float)));
    // initial weights and biases uniform in +-1/sqrt(fan_in) from a seeded host generator
    std::vector<float> p(kParams);
    std::mt19937_64 rng(seed);
    for (int l = 1; l <= 5; ++l) {
        const int nin = l == 1 ? kIn : kHid, nout = l == 5 ? kOut : kHid;
        std::uniform_real_distribution<float> U(-1.0f / std::sqrt((float)nin), 1.0f / std::sqrt((float)nin));
        for (long long i = 0; i < (long long)nin * nout; ++i) p[off_w(l) + i] = U(rng);
        for (int i = 0; i < nout; ++i) p[off_b(l) + i] = U(rng);
    }
    MCU(cudaMemcpy(m->params, p.data(), kParams * sizeof(float), cudaMemcpyHostToDevice));
    pack_kernel<<<(int)((kParams + 255) / 256), 256, 0, m->stream>>>(m->params, m->pa);
    MCU(cudaGetLastError());
    MCU(cudaStreamSynchronize(m->stream));
    *out = m;
    return CLR_OK;
}

int clr_mlp_destroy(clr_mlp* m) {
    if (!m) return CLR_ERR_INVALID_ARGUMENT;
    cudaSetDevice(m->device);
    if (m->stream) cudaStreamSynchronize(m->stream);
    if (m->step_exec) cudaGraphExecDestroy(m->step_exec);
    for (void* p : m->allocs) cudaFree(p);
    cudaFree(m->d_hp);
    if (m->ev0) cudaEventDestroy(m->ev0);
    if (m->ev1) cudaEventDestroy(m->ev1);
    if (m->fork) cudaEventDestroy(m->fork);
    if (m->join) cudaEventDestroy(m->join);
    if (m->side) cudaStreamDestroy(m->side);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
    return CLR_OK;
}

const char* clr_mlp_last_error(const clr_mlp* m) { return m ? m->err.c_str() : "null network"; }

int clr_mlp_set_params(clr_mlp* m, const float* host, int64_t count) {
    if (!m || !host || count != kParams) return mfail(m, CLR_ERR_INVALID_ARGUMENT, "expected CLR_MLP_PARAMS floats");
    MCU(cudaSetDevice(m->device));
    MCU(cudaMemcpyAsync(m->params, host, kParams * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    MCU(cudaMemsetAsync(m->m1, 0, kParams * sizeof(float), m->stream));
    MCU(cudaMemsetAsync(m->m2, 0, kParams * sizeof(float), m->stream));
    pack_kernel<<<(int)((kParams + 255) / 256), 256, 0, m->stream>>>(m->params, m->pa);
    MCU(cudaGetLastError());
    MCU(cudaStreamSynchronize(m->stream));
    m->steps = 0;
    return CLR_OK;
}

int clr_mlp_get_params(clr_mlp* m, float* host, int64_t count) {
    if (!m || !host || count != kParams) return mfail(m, CLR_ERR_INVALID_ARGUMENT, "expected CLR_MLP_PARAMS floats");
    MCU(cudaSetDevice(m->device));
    MCU(cudaMemcpyAsync(host, m->params, kParams * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    MCU(cudaStreamSynchronize(m->stream));
    return CLR_OK;
}

int clr_mlp_forward(clr_mlp* m, const float* d_x, int64_t n, float* d_y, void* stream) {
    if (!m || !d_x || !d_y || n < 0) return mfail(m, CLR_ERR_INVALID_ARGUMENT, "clr_mlp_forward: bad arguments");
    MCU(cudaSetDevice(m->device));
    cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : m->stream;
    MCU(cudaEventRecord(m->ev0, st));
    if (n > 0) {
        InferArgs a{};
        a.x = d_x; a.y = d_y; a.n = n;
        const long long tiles = (n + kM - 1) / kM;
        if (tiles > (1LL << 30)) return mfail(m, CLR_ERR_INVALID_ARGUMENT, "clr_mlp_forward: too many rows");
        a.tiles = (int)tiles;
        a.wp[0] = m->pa.wp[2]; a.wp[1] = m->pa.wp[3]; a.wp[2] = m->pa.wp[4];
        a.w1p = m->pa.wp[1]; a.w5p = m->pa.wp[5]; a.params = m->params; a.err = m->d_err;
        const int grid = (int)std::min<long long>(tiles, m->num_sms);
        mlp_infer_kernel<<<grid, kInferThreads, kInferSmem, st>>>(a);
        MCU(cudaGetLastError());
    }
    MCU(cudaEventRecord(m->ev1, st));
    MCU(cudaStreamSynchronize(st));
    MCU(cudaEventElapsedTime(&m->last_ms, m->ev0, m->ev1));
    return check_dev(m);
}

int clr_mlp_gradients(clr_mlp* m, const float* d_x, const float* d_t, int64_t n, float* grads_host, float* loss) {
    if (!m || !d_x || !d_t || n < 128 || n > m->cap || n % 128)
        return mfail(m, CLR_ERR_INVALID_ARGUMENT, "clr_mlp_gradients: n must be a multiple of 128 up to max_batch");
    MCU(cudaSetDevice(m->device));
    cudaStream_t st = m->stream;
    MCU(cudaMemsetAsync(m->loss, 0, sizeof(float), st));
    const StepArgs args = {d_x, d_t, m->d_w, nullptr, 0};
    MCU(cudaMemcpyAsync(m->d_step, &args, sizeof args, cudaMemcpyHostToDevice, st));
    MCU(forward_rows(m, (int)n, st));
    MCU(backward_rows(m, (int)n, st));
    float ls = 0.0f;
    MCU(cudaMemcpyAsync(&ls, m->loss, sizeof(float), cudaMemcpyDeviceToHost, st));
    if (grads_host) {
        sum_grads_kernel<<<(int)((kParams + 255) / 256), 256, 0, st>>>(grad_parts(m, (int)n), m->grads);
        MCU(cudaGetLastError());
        MCU(cudaMemcpyAsync(grads_host, m->grads, kParams * sizeof(float), cudaMemcpyDeviceToHost, st));
    }
    int rc = check_dev(m);
    if (rc != CLR_OK) return rc;
    if (loss) *loss = ls / (3.0f * (float)n);
    return CLR_OK;
}

}  // extern "C"

// One training step (gather, forward, backward, Adam) captured as a graph for batch size n.
static int build_step_graph(clr_mlp* m, int n) {
    if (m->step_exec && m->step_n == n) return CLR_OK;
    if (m->step_exec) {
        cudaGraphExecDestroy(m->step_exec);
        m->step_exec = nullptr;
    }
    cudaStream_t st = m->stream;
    cudaGraph_t graph;
    MCU(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    cudaError_t e = forward_rows(m, n, st);
    if (e == cudaSuccess) e = backward_rows(m, n, st);
    if (e == cudaSuccess) {
        adam_kernel<<<(int)((kParams + 255) / 256), 256, 0, st>>>(m->params, grad_parts(m, n), m->m1, m->m2, m->d_step, m->d_hp,
                                                                  m->pa);
        e = cudaGetLastError();
    }
    cudaError_t e2 = cudaStreamEndCapture(st, &graph);
    MCU(e);
    MCU(e2);
    e = cudaGraphInstantiate(&m->step_exec, graph, 0);
    cudaGraphDestroy(graph);
    MCU(e);
    m->step_n = n;
    return CLR_OK;
}

extern "C" int clr_mlp_train(clr_mlp* m, const float* d_x, const float* d_t, const int32_t* d_index, int64_t n_index,
                             int batch, float lr, float* mean_loss) {
    if (!m || !d_x || !d_t || !d_index || batch < 128 || batch % 128 || batch > m->cap || n_index < batch)
        return mfail(m, CLR_ERR_INVALID_ARGUMENT,
                     "clr_mlp_train: batch must be a multiple of 128 up to max_batch, and at most n_index");
    MCU(cudaSetDevice(m->device));
    cudaStream_t st = m->stream;
    const long long steps = n_index / batch;
    if (steps > m->hp_cap) {  // the captured step holds the old address
        if (m->step_exec) cudaGraphExecDestroy(m->step_exec);
        m->step_exec = nullptr;
        cudaFree(m->d_hp);
        m->d_hp = nullptr;
        m->hp_cap = 0;
        const long long cap = std::max(2 * steps, 256LL);
        MCU(cudaMalloc((void**)&m->d_hp, (size_t)cap * sizeof(float4)));
        m->hp_cap = cap;
    }
    int rc = build_step_graph(m, batch);
    if (rc != CLR_OK) return rc;
    std::vector<float4> hp(steps);
    for (long long s = 0; s < steps; ++s) {
        m->steps++;
        hp[s] = make_float4(lr, 1.0f - std::pow(0.9f, (float)m->steps), 1.0f - std::pow(0.999f, (float)m->steps), 0.0f);
    }
    const StepArgs args = {d_x, d_t, m->d_w, d_index, 0};
    // pageable copies are staged by the driver before the calls return
    MCU(cudaMemcpyAsync(m->d_step, &args, sizeof args, cudaMemcpyHostToDevice, st));
    MCU(cudaMemcpyAsync(m->d_hp, hp.data(), (size_t)steps * sizeof(float4), cudaMemcpyHostToDevice, st));
    MCU(cudaMemsetAsync(m->loss, 0, sizeof(float), st));
    MCU(cudaEventRecord(m->ev0, st));
    for (long long s = 0; s < steps; ++s) MCU(cudaGraphLaunch(m->step_exec, st));
    MCU(cudaEventRecord(m->ev1, st));
    float ls = 0.0f;
    MCU(cudaMemcpyAsync(&ls, m->loss, sizeof(float), cudaMemcpyDeviceToHost, st));
    rc = check_dev(m);
    if (rc != CLR_OK) return rc;
    MCU(cudaEventElapsedTime(&m->last_ms, m->ev0, m->ev1));
    if (mean_loss) *mean_loss = steps > 0 ? ls / (3.0f * (float)batch * (float)steps) : 0.0f;
    return CLR_OK;
}

extern "C" int clr_mlp_set_loss_weights(clr_mlp* m, const float* d_w) {
    if (!m) return CLR_ERR_INVALID_ARGUMENT;
    m->d_w = d_w;
    return CLR_OK;
}

extern "C" int clr_mlp_last_ms(const clr_mlp* m, float* ms) {
    if (!m || !ms) return CLR_ERR_INVALID_ARGUMENT;
    *ms = m->last_ms;
    return CLR_OK;
}

// Plain tensor-core product C[M][256] = A[M][K] . B[256][K]^T (BF16 in, FP32 out), the kernel the
// network's layers use, exposed for its own tests and for callers with other 256-wide products.
extern "C" int clr_bf16_gemm_n256(const void* d_a, int64_t lda, const void* d_b, int64_t ldb, int64_t M, int64_t K,
                                  float* d_c, int64_t ldc, void* stream) {
    if (!d_a || !d_b || !d_c || M < 1 || K < 64 || K % 64 || lda % 8 || ldb % 8 || ldc % 4 || lda < K || ldb < K ||
        ldc < 256 || (reinterpret_cast<uintptr_t>(d_a) & 15) || (reinterpret_cast<uintptr_t>(d_b) & 15) ||
        (reinterpret_cast<uintptr_t>(d_c) & 15))
        return CLR_ERR_INVALID_ARGUMENT;
    static int* err = nullptr;  // error word of this entry point (first device it runs on)
    if (!err && cudaMalloc(&err, sizeof(int)) != cudaSuccess) return CLR_ERR_CUDA;
    if (set_gemm_attributes() != cudaSuccess) return CLR_ERR_CUDA;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(err, 0, sizeof(int), st) != cudaSuccess) return CLR_ERR_CUDA;
    GemmBatch b{};
    GemmArgs& g = b.g[0];
    g.A = static_cast<const bf16*>(d_a); g.lda = lda; g.B = static_cast<const bf16*>(d_b); g.ldb = ldb;
    g.M = (int)M; g.K = (int)K; g.k_split = (int)K; g.out_f32 = d_c; g.ldo = ldc; g.err = err;
    const bool wide = (M + kM - 1) / kM >= kWideTiles;
    if ((wide ? launch_gemm<EPI_STORE_F32, kN>(b, 1, 1, st) : launch_gemm<EPI_STORE_F32>(b, 1, 1, st)) != cudaSuccess)
        return CLR_ERR_CUDA;
    int herr = 0;
    if (cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess) return CLR_ERR_CUDA;
    if (cudaStreamSynchronize(st) != cudaSuccess) return CLR_ERR_CUDA;
    return herr ? CLR_ERR_DEVICE_TIMEOUT : CLR_OK;
}

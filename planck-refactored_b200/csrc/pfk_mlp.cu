// pfk_mlp.cu -- the learned-guess network: a small multilayer perceptron
// trained and evaluated by this file's kernels on the GPU.
//
//   H_0 = bf16(X);  Z_l = H_{l-1} W_l + b_l;  H_l = bf16(SiLU(Z_l)) (l < L);
//   Y = Z_L (FP32).
//
// Every matrix product runs on the fifth-generation tensor cores as BF16 x
// BF16 with FP32 accumulation in tensor memory (tcgen05.mma, M 128, N 64,
// K 16); weights are kept in FP32 (Adam's master copy) and rounded to BF16
// for the products.  Training minimises the mean
// squared error against targets T with Adam.  The backward pass:
//   dZ_L = 2 (Y - T) / (n d_L);  dW_l = H_{l-1}^T bf16(dZ_l);
//   db_l = column sums of dZ_l;  dH_{l-1} = bf16(dZ_l) W_l^T;
//   dZ_{l-1} = dH_{l-1} * SiLU'(Z_{l-1}).
//
// Networks up to 256 wide run a training step in three launches: everything
// up to dZ_1 (fused_kernel), the weight gradients of every layer, and the
// update.  Wider ones take 2L + 2 for L layers: the input conversion, L
// forward products (the last one also forms dZ_L and the loss), L - 1
// products for dH (their epilogue applies SiLU' and leaves dZ), and the same
// last two.  Each product
// leaves its result in both orders (rows of the batch, and transposed), so
// every product reads both operands as rows of K by 16-byte copies.  On the
// 112-256-256-232 network (one B200): 2048 rows, a step 89 us against 1675 us
// before (products staged by 2-byte gathers, bias sums by one thread per
// column, weight gradients on 8 CTAs, two host synchronisations); forward of
// 8192 rows 47 us against 250 us (both with the host call).
// The reference has no counterpart: it is the learned part of the guess
// hook (scf.cpp:206-240 selects the guess; a learned density enters the SCF
// as a ReadDensity guess does, scf.cpp:213-216).
#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "planck_fock.h"

namespace {

thread_local std::string g_mlp_error;

// ---------------------------------------------------------------------------
// GEMM on the fifth-generation tensor cores: acc[m][n] = sum_k A[m][k] B[n][k]
// with both operands stored as rows of K (BF16, row strides lda and ldb, every
// row start 16-byte aligned), FP32 accumulation in tensor memory, and one of
// the epilogues below.
//
// One CTA of 512 threads per 128 x 64 tile.  K goes in rounds of 64 through a
// ring of TC_STAGES shared-memory stages: cp.async copies 16-byte segments of
// later rounds while the tensor cores work on the current one (the products
// here are 2 to 64 rounds deep, so a tile's time is the latency of its loads;
// the ring keeps three rounds in flight).  Stages hold the operands K-major in
// the no-swizzle core-matrix layout (8 rows x 16 bytes per 128-byte core
// matrix), zero-filled outside the matrices; a warp's copies cover 8 rows x 4
// segments, which is 64 contiguous bytes per row in global memory and 512
// contiguous bytes in shared memory.  One thread issues four tcgen05.mma
// (M 128, N 64, K 16) per round and commits them to the stage's mbarrier,
// which every thread waits on before it refills the stage.  The epilogue reads
// the accumulator back with tcgen05.ld, warps w, w + 4, w + 8 and w + 12 taking
// rows 32w .. 32w+31 (the tensor-memory lanes a warp may access) and 16 columns
// each: a tile's time is mostly this epilogue, a latency-bound chain per
// thread, so it is spread over 16 warps (with 4 warps the three layers'
// forward pass of 8192 rows took 73 us, with 8 and overlapped launches 54).
// Waits are bounded (2 s of
// SM cycles); a wait that runs out sets *err, the CTA stops issuing, waits
// (bounded again) for what is in flight and frees its columns.
// ---------------------------------------------------------------------------
constexpr int TC_M = 128, TC_N = 64, TC_K = 64, TC_STAGES = 4, TC_THREADS = 512;
constexpr int TC_A_BYTES = TC_M * TC_K * 2, TC_B_BYTES = TC_N * TC_K * 2, TC_STAGE_BYTES = TC_A_BYTES + TC_B_BYTES;
// 96 KB of stages: two CTAs share an SM, and their 2 x 64 accumulator columns
// fit its 512 tensor-memory columns
constexpr int TC_SMEM = TC_STAGES * TC_STAGE_BYTES;
constexpr uint32_t TC_TMEM_COLS = 64;
constexpr long long TC_WAIT_CYCLES = 4000000000ll;   // 2 s at 1.965 GHz
// instruction descriptor (kind::f16): D F32 (bits 4-5 = 1), A and B BF16
// (bits 7-9 = 1, 10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3 at bits
// 17-22, M >> 4 at bits 24-28
constexpr uint32_t TC_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TC_N >> 3) << 17) |
                              ((uint32_t)(TC_M >> 4) << 24);
constexpr int kMaxLayers = 8;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Byte offset of the 16-byte segment (row, K chunk kc of 8 elements) in a
// staged tile: K chunks of a row group are adjacent core matrices (128 B
// apart), row groups of 8 are TC_K / 8 core matrices apart.
__device__ __forceinline__ uint32_t tc_off(int row, int kc)
{
    return (uint32_t)(((row >> 3) * (TC_K / 8) + kc) * 128 + (row & 7) * 16);
}

// Shared-memory matrix descriptor of a K-major, no-swizzle operand whose
// first core matrix is at saddr: leading byte offset 128 (the next K chunk),
// stride byte offset TC_K / 8 * 128 (the next group of 8 rows), descriptor
// version 1 (bit 46), base offset 0, layout type 0 (no swizzle).
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr)
{
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(128u >> 4) << 16) |
           ((uint64_t)((TC_K / 8 * 128u) >> 4) << 32) | (1ull << 46);
}

// Waits until phase `parity` of the mbarrier at bar completes; false after
// TC_WAIT_CYCLES SM cycles without completion.
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity)
{
    const long long t0 = clock64();
    while (true) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (done) return true;
        if (clock64() - t0 > TC_WAIT_CYCLES) return false;
    }
}

__device__ __forceinline__ unsigned pack2(__nv_bfloat16 lo, __nv_bfloat16 hi)
{
    return (unsigned)__bfloat16_as_ushort(lo) | ((unsigned)__bfloat16_as_ushort(hi) << 16);
}

__device__ __forceinline__ float silu(float z) { return z / (1.0f + __expf(-z)); }
__device__ __forceinline__ float silu_grad(float z)
{
    const float s = 1.0f / (1.0f + __expf(-z));
    return s * (1.0f + z * (1.0f - s));
}

// Programmatic dependent launch: a kernel launched with launch_after may start
// while its predecessor in the stream finishes; grid_wait returns when that
// one has completed and its writes are visible, grid_launch_next lets the
// successor start.  A step is a chain of kernels of a few microseconds each,
// so the launch gaps are a good part of it.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
void launch_after(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);   // a failure shows in cudaGetLastError
}

// Copies a 16-byte segment to shared memory asynchronously; zero fill when !ok.
__device__ __forceinline__ void cp16(uint32_t dst, const void *src, bool ok)
{
    const int n = ok ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

// One round of an operand tile: rows row0 .. row0 + ROWS - 1, K columns
// k0 .. k0 + TC_K - 1, zero outside row < nrows and k < kend (kend a multiple
// of 8, or the storage behind it zero up to the next one).
template <int ROWS>
__device__ __forceinline__ void tc_load(uint32_t sbase, const __nv_bfloat16 *__restrict__ src, long long ld, int row0,
                                        int nrows, int k0, int kend)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < ROWS / 4 / (TC_THREADS / 32); ++i) {
        // unit u: rows 8 (u >> 1) .. + 7, segments 4 (u & 1) .. + 3
        const int u = i * (TC_THREADS / 32) + warp;
        const int r = (u >> 1) * 8 + (lane & 7), kc = (u & 1) * 4 + (lane >> 3);
        const int gr = row0 + r, gk = k0 + kc * 8;
        const bool ok = gr < nrows && gk < kend;
        cp16(sbase + tc_off(r, kc), ok ? src + (size_t)gr * ld + gk : src, ok);
    }
}

// Epilogues.  kEpiHidden: x = acc + bias; Z = x and its transposed SiLU when
// training, H = bf16(SiLU(x)).  kEpiOut: Y = acc + bias.  kEpiLoss: r = acc +
// bias - T, d = 2 r scale: G, its transpose, column sums of d, sum of r^2
// scale.  kEpiBack: d = acc SiLU'(Z): G, its transpose, column sums.
// kEpiPart: the tile itself (a part of the sum over K).
enum { kEpiHidden, kEpiOut, kEpiLoss, kEpiBack, kEpiPart };

struct EpiArgs {
    const float *bias;        // per column
    float *Z;                 // pre-activations (written: hidden, training; read: back), row stride N
    const float *T;           // targets, row stride N
    float *Y;                 // output, row stride N
    __nv_bfloat16 *R, *RT;    // result rows (stride N; null: not wanted) and transposed (row stride ldt; null: not wanted)
    long long ldt;
    float *colpart;           // column sums per row tile: [row tile][N]
    double *losspart;         // per tile
    float scale;
    bool vec;                 // T or Y is 16-byte aligned
};

// Sum over the warp's 32 lanes of each of v[0..15]: lane 2c and 2c + 1 return
// column c's (each step keeps half of the columns and adds the partner
// lane's halves: 16 shuffles instead of 80).
__device__ __forceinline__ float colsum16(const float (&v)[16], int lane)
{
    float a[8], b[4], c[2], d;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const bool up = lane & 16;
        a[i] = (up ? v[i + 8] : v[i]) + __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + 8], 16);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const bool up = lane & 8;
        b[i] = (up ? a[i + 4] : a[i]) + __shfl_xor_sync(0xffffffffu, up ? a[i] : a[i + 4], 8);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const bool up = lane & 4;
        c[i] = (up ? b[i + 2] : b[i]) + __shfl_xor_sync(0xffffffffu, up ? b[i] : b[i + 2], 4);
    }
    {
        const bool up = lane & 2;
        d = (up ? c[1] : c[0]) + __shfl_xor_sync(0xffffffffu, up ? c[0] : c[1], 2);
    }
    return d + __shfl_xor_sync(0xffffffffu, d, 1);
}

// The epilogue of the tile at (m0, n0) of an M x N result, from the
// accumulator at tmem (zero when !have).  bias: the tile's columns; colw and
// lossw: shared scratch; part: the tile's FP32 destination (kEpiPart).
template <int EPI>
__device__ __forceinline__ void tile_epilogue(uint32_t tmem, bool have, int M, int N, int m0, int n0, const EpiArgs &e,
                                              const float *bias, float (*colw)[TC_N], double *lossw, float *part)
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int quad = warp & 3, m = m0 + quad * 32 + lane;
    constexpr int kCols = TC_N / (TC_THREADS / 128);   // per warp
    static_assert(kCols % 16 == 0, "a warp reads 16 columns at a time");
    const int c0 = (warp >> 2) * kCols;
    double loss = 0.0;
#pragma unroll 1
    for (int c = c0; c < c0 + kCols; c += 16) {
        uint32_t v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = 0u;
        if (have) {
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
                         "%11, %12, %13, %14, %15}, [%16];"
                         : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                           "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                           "=r"(v[14]), "=r"(v[15])
                         : "r"(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)c));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        }
        if constexpr (EPI == kEpiPart) {
            float4 *o = reinterpret_cast<float4 *>(part + (size_t)(quad * 32 + lane) * TC_N + c);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                o[i] = make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]),
                                   __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3]));
        } else {
            // widths are multiples of 8: each half of the 16 columns is inside or outside
            float x[16];
            __nv_bfloat16 h[16];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int n = n0 + c + 8 * half;
                const bool in = m < M && n < N;
                const size_t at = (size_t)m * N + n;
                float t[8] = {};
                if (EPI == kEpiLoss && in) {
                    if (e.vec) {
                        *reinterpret_cast<float4 *>(t) = __ldg(reinterpret_cast<const float4 *>(e.T + at));
                        *reinterpret_cast<float4 *>(t + 4) = __ldg(reinterpret_cast<const float4 *>(e.T + at + 4));
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; ++i) t[i] = __ldg(e.T + at + i);
                    }
                }
                if (EPI == kEpiBack && in) {
                    *reinterpret_cast<float4 *>(t) = *reinterpret_cast<const float4 *>(e.Z + at);
                    *reinterpret_cast<float4 *>(t + 4) = *reinterpret_cast<const float4 *>(e.Z + at + 4);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int k = 8 * half + i;
                    float a = __uint_as_float(v[k]);
                    if (EPI != kEpiBack) a += bias[c + k];
                    if (EPI == kEpiLoss) {
                        const float r = a - t[i];
                        if (in) loss += (double)r * r * e.scale;
                        a = 2.0f * r * e.scale;
                    }
                    if (EPI == kEpiBack) a *= silu_grad(t[i]);
                    x[k] = in ? a : 0.0f;
                    if (EPI == kEpiHidden) h[k] = in ? __float2bfloat16(silu(a)) : __float2bfloat16(0.0f);
                    if (EPI == kEpiLoss || EPI == kEpiBack) h[k] = __float2bfloat16(x[k]);
                }
                if ((EPI == kEpiHidden && e.Z) || EPI == kEpiOut) {
                    float *o = EPI == kEpiOut ? e.Y : e.Z;
                    if (in) {
                        if (EPI == kEpiHidden || e.vec) {
                            *reinterpret_cast<float4 *>(o + at) = *reinterpret_cast<const float4 *>(x + 8 * half);
                            *reinterpret_cast<float4 *>(o + at + 4) = *reinterpret_cast<const float4 *>(x + 8 * half + 4);
                        } else {
#pragma unroll
                            for (int i = 0; i < 8; ++i) o[at + i] = x[8 * half + i];
                        }
                    }
                }
                if (EPI != kEpiOut) {
                    if (e.R && in) {
                        uint4 w;
                        w.x = pack2(h[8 * half], h[8 * half + 1]);
                        w.y = pack2(h[8 * half + 2], h[8 * half + 3]);
                        w.z = pack2(h[8 * half + 4], h[8 * half + 5]);
                        w.w = pack2(h[8 * half + 6], h[8 * half + 7]);
                        *reinterpret_cast<uint4 *>(e.R + at) = w;
                    }
                    // transposed, zero up to the next multiple of 8 rows: the
                    // weight-gradient products read whole 16-byte segments
                    if (e.RT && n < N && m < ((M + 7) & ~7)) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) e.RT[(size_t)(n + i) * e.ldt + m] = h[8 * half + i];
                    }
                }
            }
            if constexpr (EPI == kEpiLoss || EPI == kEpiBack) {
                const float s = colsum16(x, lane);
                if (!(lane & 1)) colw[quad][c + (lane >> 1)] = s;
            }
        }
    }
    if constexpr (EPI == kEpiLoss || EPI == kEpiBack) {
        if (EPI == kEpiLoss) {
            for (int o = 16; o; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
            if (lane == 0) lossw[warp] = loss;
        }
        __syncthreads();
        if (tid < TC_N && n0 + tid < N)
            e.colpart[(size_t)(m0 / TC_M) * N + n0 + tid] =
                (colw[0][tid] + colw[1][tid]) + (colw[2][tid] + colw[3][tid]);
        if (EPI == kEpiLoss && tid == 0) {
            double sum = 0.0;
            for (int w = 0; w < TC_THREADS / 32; ++w) sum += lossw[w];
            e.losspart[m0 / TC_M * ((N + TC_N - 1) / TC_N) + n0 / TC_N] = sum;
        }
    }
}

// The whole tile: K loop and epilogue.  part: the tile's FP32 destination (kEpiPart).
template <int EPI>
__device__ __forceinline__ void gemm_tile(int M, int N, int kbeg, int kend, const __nv_bfloat16 *__restrict__ A,
                                          long long lda, const __nv_bfloat16 *__restrict__ B, long long ldb, int m0,
                                          int n0, const EpiArgs &e, float *part, int *err)
{
    extern __shared__ __align__(128) unsigned char tc_tiles[];
    __shared__ __align__(8) unsigned long long mbar[TC_STAGES];
    __shared__ uint32_t tmem_slot;
    __shared__ float colw[4][TC_N];
    __shared__ double lossw[TC_THREADS / 32];
    __shared__ float bias[TC_N];
    const int tid = threadIdx.x, warp = tid >> 5;
    const uint32_t s0 = smem_u32(tc_tiles), sbar = smem_u32(mbar);
    const int nk = kend > kbeg ? (kend - kbeg + TC_K - 1) / TC_K : 0;
    auto load = [&](int kt) {
        if (kt < nk) {
            const uint32_t st = s0 + (kt % TC_STAGES) * TC_STAGE_BYTES;
            tc_load<TC_M>(st, A, lda, m0, M, kbeg + kt * TC_K, kend);
            tc_load<TC_N>(st + TC_A_BYTES, B, ldb, n0, N, kbeg + kt * TC_K, kend);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");   // one group per round, empty past the end
    };
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(TC_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < TC_STAGES; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sbar + 8 * i) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // everything above overlaps the previous kernel's end; its results are
    // read only from here on
    grid_wait();
    grid_launch_next();
#pragma unroll
    for (int i = 0; i < TC_STAGES - 1; ++i) load(i);
    if (EPI != kEpiPart && EPI != kEpiBack && tid < TC_N) bias[tid] = n0 + tid < N ? e.bias[n0 + tid] : 0.0f;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;

    bool failed = false;
    int issued = 0;
    for (int kt = 0; kt < nk; ++kt) {
        bool ok = true;
        // round kt + TC_STAGES - 1 reuses the stage of round kt - 1
        if (kt > 0 && kt + TC_STAGES - 1 < nk)
            ok = tc_wait(sbar + 8 * ((kt - 1) % TC_STAGES), ((kt - 1) / TC_STAGES) & 1);
        if (ok) load(kt + TC_STAGES - 1);
        asm volatile("cp.async.wait_group %0;" ::"n"(TC_STAGES - 1) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // staged tiles visible to the tensor cores
        if (__syncthreads_or(!ok)) {
            failed = true;
            break;
        }
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t st = s0 + (kt % TC_STAGES) * TC_STAGE_BYTES;
#pragma unroll
            for (int s = 0; s < TC_K / 16; ++s) {
                const uint64_t da = tc_desc(st + s * 256), db = tc_desc(st + TC_A_BYTES + s * 256);
                const uint32_t accumulate = (kt > 0 || s > 0) ? 1u : 0u;
                asm volatile("{\n\t.reg .pred p;\n\t"
                             "setp.ne.b32 p, %4, 0;\n\t"
                             "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
                             "l"(da), "l"(db), "r"(TC_IDESC), "r"(accumulate)
                             : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             sbar + 8 * (kt % TC_STAGES))
                         : "memory");
        }
        ++issued;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    // the last commit tracks every product before it
    if (issued > 0) {
        const bool ok = tc_wait(sbar + 8 * ((issued - 1) % TC_STAGES), ((issued - 1) / TC_STAGES) & 1);
        if (__syncthreads_or(!ok)) {
            failed = true;
            // once more (bounded) before the accumulator columns are released below
            tc_wait(sbar + 8 * ((issued - 1) % TC_STAGES), ((issued - 1) / TC_STAGES) & 1);
        }
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    if (failed) {
        if (tid == 0) {
            *(volatile int *)err = 1;
            __threadfence_system();
        }
    } else {
        tile_epilogue<EPI>(tmem, nk > 0, M, N, m0, n0, e, bias, colw, lossw, part);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TC_TMEM_COLS) : "memory");
}

template <int EPI>
__global__ void __launch_bounds__(TC_THREADS, 2) gemm_tc_kernel(int M, int N, int K, const __nv_bfloat16 *__restrict__ A,
                                                      const __nv_bfloat16 *__restrict__ B, EpiArgs e, int *err)
{
    gemm_tile<EPI>(M, N, 0, K, A, K, B, K, blockIdx.y * TC_M, blockIdx.x * TC_N, e, nullptr, err);
}

// The layers as the gradient kernels see them.
struct Layers {
    int nl, splits, tiles;                 // tiles: 128 x 64 tiles of all weight matrices
    int ksplit;                            // batch rows per split (a multiple of TC_K)
    int din[kMaxLayers], dout[kMaxLayers], tile0[kMaxLayers];
    long long w_off[kMaxLayers], b_off[kMaxLayers], col_off[kMaxLayers];
    const __nv_bfloat16 *HT[kMaxLayers], *GT[kMaxLayers];
};

// Weight gradients of every layer in one launch: CTA (tile, split) sums its
// 128 x 64 tile of dW_l = H^T G over its share of the batch.  A layer alone is
// 4 to 8 tiles of 2048 rows on a 148-SM chip; all layers' tiles times the
// splits fill it, and the update adds the parts in a fixed order.
__global__ void __launch_bounds__(TC_THREADS, 2) gemm_dw_kernel(Layers L, int n, long long ldt, float *part, int *err)
{
    int l = 0;
    while (l + 1 < L.nl && (int)blockIdx.x >= L.tile0[l + 1]) ++l;
    const int tile = blockIdx.x - L.tile0[l], tn = (L.dout[l] + TC_N - 1) / TC_N;
    const int k0 = blockIdx.y * L.ksplit, k1 = min(n, k0 + L.ksplit);
    EpiArgs e{};
    gemm_tile<kEpiPart>(L.din[l], L.dout[l], k0, k1, L.HT[l], ldt, L.GT[l], ldt, tile / tn * TC_M, tile % tn * TC_N, e,
                        part + ((size_t)blockIdx.y * L.tiles + blockIdx.x) * (TC_M * TC_N), err);
}

// H = bf16(X) and, with HT, its transpose (zero up to the next multiple of 8
// rows); 32 x 32 tiles through shared memory, rows of the batch along grid.x
// (grid.y ends at 65535).
__global__ void __launch_bounds__(256) input_kernel(const float *__restrict__ X, int n, int d, __nv_bfloat16 *H,
                                                    __nv_bfloat16 *HT, long long ldt)
{
    __shared__ __nv_bfloat16 tile[32][33];
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5, c0 = blockIdx.y * 32, r0 = blockIdx.x * 32;
    grid_launch_next();
#pragma unroll
    for (int i = y; i < 32; i += 8) {
        const int r = r0 + i, c = c0 + x;
        const bool in = r < n && c < d;
        const __nv_bfloat16 v = __float2bfloat16(in ? X[(size_t)r * d + c] : 0.0f);
        if (in) H[(size_t)r * d + c] = v;
        tile[i][x] = v;
    }
    if (!HT) return;
    __syncthreads();
#pragma unroll
    for (int i = y; i < 32; i += 8) {
        const int r = r0 + x, c = c0 + i;
        if (c < d && r < ((n + 7) & ~7)) HT[(size_t)c * ldt + r] = tile[x][i];
    }
}

// BF16 weights in both orders (rows of din, rows of dout) from the FP32 ones.
__global__ void weights_kernel(const float *__restrict__ p, Layers L, __nv_bfloat16 *wb, __nv_bfloat16 *wt)
{
    const int l = blockIdx.y, din = L.din[l], dout = L.dout[l];
    const long long nw = (long long)din * dout;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nw; i += (long long)gridDim.x * blockDim.x) {
        const __nv_bfloat16 w = __float2bfloat16(p[L.w_off[l] + i]);
        wb[L.w_off[l] + i] = w;
        wt[L.w_off[l] + (i % dout) * din + i / dout] = w;
    }
}

struct AdamArgs {
    float lr, b1, b2, eps, c1, c2;
};

// Gradient of every parameter (the parts of dW, the row tiles' column sums of
// dZ for the biases, each added in order), then Adam (bias-corrected) on the
// FP32 parameters and the BF16 weights of the next forward pass; with UPDATE
// false the gradient vector instead.  Block (0, 0) adds up the loss and
// leaves it where the host reads it.
template <bool UPDATE>
__global__ void __launch_bounds__(256) update_kernel(Layers L, const float *__restrict__ part,
                                                     const float *__restrict__ colpart, int row_tiles,
                                                     const double *__restrict__ losspart, int nloss, double *loss_out,
                                                     float *__restrict__ grad, float *__restrict__ p,
                                                     float *__restrict__ m, float *__restrict__ v, __nv_bfloat16 *wb,
                                                     __nv_bfloat16 *wt, AdamArgs a)
{
    const int l = blockIdx.y, din = L.din[l], dout = L.dout[l];
    const int tn = (dout + TC_N - 1) / TC_N;
    grid_wait();
    const long long nw = (long long)din * dout, n = nw + dout;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float g = 0.0f;
        int r = 0, c = 0;
        if (i < nw) {
            r = (int)(i / dout);
            c = (int)(i % dout);
            const float *q = part + (size_t)(L.tile0[l] + (r / TC_M) * tn + c / TC_N) * (TC_M * TC_N) +
                             (r % TC_M) * TC_N + c % TC_N;
#pragma unroll 8
            for (int s = 0; s < L.splits; ++s) g += q[(size_t)s * L.tiles * (TC_M * TC_N)];
        } else {
#pragma unroll 8
            for (int t = 0; t < row_tiles; ++t) g += colpart[L.col_off[l] + (size_t)t * dout + (i - nw)];
        }
        const long long at = i < nw ? L.w_off[l] + i : L.b_off[l] + (i - nw);
        if constexpr (UPDATE) {
            const float mi = a.b1 * m[at] + (1.0f - a.b1) * g, vi = a.b2 * v[at] + (1.0f - a.b2) * g * g;
            m[at] = mi;
            v[at] = vi;
            const float w = p[at] - a.lr * (mi * a.c1) / (sqrtf(vi * a.c2) + a.eps);
            p[at] = w;
            if (i < nw) {
                wb[at] = __float2bfloat16(w);
                wt[L.w_off[l] + (long long)c * din + r] = __float2bfloat16(w);
            }
        } else {
            grad[at] = g;
        }
    }
    if (blockIdx.x == 0 && blockIdx.y == 0) {
        __shared__ double part_sum[256];
        double s = 0.0;
        for (int i = threadIdx.x; i < nloss; i += 256) s += losspart[i];
        part_sum[threadIdx.x] = s;
        __syncthreads();
        for (int o = 128; o; o >>= 1) {
            if (threadIdx.x < (unsigned)o) part_sum[threadIdx.x] += part_sum[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) *loss_out = part_sum[0];
    }
}

unsigned blocks_for(long long n) { return (unsigned)std::min<long long>((n + 255) / 256, 148 * 16); }

// All layers of a network whose widths are at most kFuseWidth in one kernel: a
// cluster of four CTAs takes 128 rows of the batch through the forward pass
// (with TRAIN also the loss and the backward pass to dZ_1), CTA c computing
// columns 64c .. 64c + 63 of every layer.  A layer of 128 rows is a microsecond
// of loads and products and two of epilogue; as a launch of its own it took 8
// to 10.  Between layers the CTAs exchange their columns through global
// memory (L2) and a cluster barrier; the next layer's weights are fetched
// while the epilogue runs.  The layer's whole K (at most four rounds) sits in
// the four stages.  Every CTA passes every barrier, also one whose wait ran out.
// 112-256-256-232, 2048 rows: a step 98 -> 89 us, forward of 8192 rows 54 ->
// 47 us (with 16-warp epilogues and waits that poll the SM clock instead of
// the global timer).
constexpr int kFuseWidth = 256, kFuseCtas = 4;
static_assert(kFuseWidth <= TC_STAGES * TC_K && kFuseWidth <= kFuseCtas * TC_N, "a layer must fit the stages and the cluster");

struct FusedArgs {
    int n, nl;
    int dims[kMaxLayers + 1];
    const float *X, *T;
    float *Y;
    const __nv_bfloat16 *wt[kMaxLayers], *wb[kMaxLayers];
    const float *bias[kMaxLayers];
    float *Z[kMaxLayers];
    __nv_bfloat16 *H[kMaxLayers], *HT[kMaxLayers], *G[kMaxLayers], *GT[kMaxLayers];
    float *colpart[kMaxLayers];
    double *losspart;
    long long ldt;
    float scale;
    bool xvec, ovec;          // X, and T or Y, are 16-byte aligned
};

__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

template <bool TRAIN>
__global__ void __launch_bounds__(TC_THREADS, TRAIN ? 1 : 2) __cluster_dims__(kFuseCtas, 1, 1) fused_kernel(FusedArgs a, int *err)
{
    extern __shared__ __align__(128) unsigned char tc_tiles[];
    __shared__ __align__(8) unsigned long long mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ float colw[4][TC_N];
    __shared__ double lossw[TC_THREADS / 32];
    __shared__ float bias[TC_N];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t s0 = smem_u32(tc_tiles), sbar = smem_u32(&mbar);
    const int m0 = blockIdx.y * TC_M, n0 = blockIdx.x * TC_N, L = a.nl;
    const int steps = TRAIN ? 2 * L - 1 : L;   // L forward layers, then dH of layers L - 1 .. 1

    // step i: forward of layer i, or (i >= L) dH of layer 2 L - 1 - i
    auto layer = [&](int i) { return i < L ? i : 2 * L - 1 - i; };
    auto width = [&](int i) { return i < L ? a.dims[i + 1] : a.dims[layer(i)]; };
    auto depth = [&](int i) { return i < L ? a.dims[i] : a.dims[layer(i) + 1]; };
    auto load_b = [&](int i) {
        const int K = depth(i), N = width(i);
        if (n0 >= N) return;
        const __nv_bfloat16 *B = i < L ? a.wt[i] : a.wb[layer(i)];
        for (int k = 0; k < K; k += TC_K)
            tc_load<TC_N>(s0 + k / TC_K * TC_STAGE_BYTES + TC_A_BYTES, B, K, n0, N, k, K);
    };
    load_b(0);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(TC_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sbar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    grid_launch_next();
    // the network's input, rounded to BF16 in place; CTA c also leaves every
    // fourth group of 8 columns transposed for the weight gradients
    {
        const int d0 = a.dims[0], rounds = (d0 + TC_K - 1) / TC_K;
        for (int u = warp; u < rounds * (TC_M / 4); u += TC_THREADS / 32) {
            const int kt = u / (TC_M / 4), v = u % (TC_M / 4);
            const int r = (v >> 1) * 8 + (lane & 7), kc = (v & 1) * 4 + (lane >> 3);
            const int gr = m0 + r, gk = kt * TC_K + kc * 8;
            const bool ok = gr < a.n && gk < d0;
            float x[8] = {};
            if (ok) {
                const float *src = a.X + (size_t)gr * d0 + gk;
                if (a.xvec) {
                    *reinterpret_cast<float4 *>(x) = __ldg(reinterpret_cast<const float4 *>(src));
                    *reinterpret_cast<float4 *>(x + 4) = __ldg(reinterpret_cast<const float4 *>(src) + 1);
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) x[i] = __ldg(src + i);
                }
            }
            __nv_bfloat16 h[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) h[i] = __float2bfloat16(x[i]);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(s0 + kt * TC_STAGE_BYTES + tc_off(r, kc)),
                         "r"(pack2(h[0], h[1])), "r"(pack2(h[2], h[3])), "r"(pack2(h[4], h[5])), "r"(pack2(h[6], h[7]))
                         : "memory");
            if (TRAIN && (gk >> 3) % kFuseCtas == (int)blockIdx.x && gk < d0 && gr < ((a.n + 7) & ~7)) {
#pragma unroll
                for (int i = 0; i < 8; ++i) a.HT[0][(size_t)(gk + i) * a.ldt + gr] = h[i];
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;

    bool failed = false;
    uint32_t parity = 0;
    for (int i = 0; i < steps; ++i) {
        const int l = layer(i), K = depth(i), N = width(i);
        const bool mine = n0 < N && !failed;   // uniform over the CTA
        const __nv_bfloat16 *A = i < L ? a.H[l] : a.G[l];
        if (mine) {
            if (i > 0)
                for (int k = 0; k < K; k += TC_K)
                    tc_load<TC_M>(s0 + k / TC_K * TC_STAGE_BYTES, A, K, m0, a.n, k, K);
            if (i < L && tid < TC_N) bias[tid] = n0 + tid < N ? a.bias[l][n0 + tid] : 0.0f;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // staged tiles visible to the tensor cores
        __syncthreads();
        if (mine) {
            if (tid == 0) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int k = 0; k < K; k += 16) {
                    const uint32_t st = s0 + k / TC_K * TC_STAGE_BYTES + k % TC_K / 16 * 256;
                    const uint64_t da = tc_desc(st), db = tc_desc(st + TC_A_BYTES);
                    const uint32_t accumulate = k > 0 ? 1u : 0u;
                    asm volatile("{\n\t.reg .pred p;\n\t"
                                 "setp.ne.b32 p, %4, 0;\n\t"
                                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
                                 "l"(da), "l"(db), "r"(TC_IDESC), "r"(accumulate)
                                 : "memory");
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(sbar)
                             : "memory");
            }
            const bool ok = tc_wait(sbar, parity);
            if (__syncthreads_or(!ok)) {
                failed = true;
                tc_wait(sbar, parity);   // once more (bounded) before the tiles and columns are used again
                if (tid == 0) {
                    *(volatile int *)err = 1;
                    __threadfence_system();
                }
            }
            parity ^= 1u;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        if (i + 1 < steps && !failed) load_b(i + 1);   // this layer's weights are used up
        if (mine && !failed) {
            EpiArgs e{};
            e.ldt = a.ldt;
            if (i + 1 < L) {
                e.Z = TRAIN ? a.Z[l] : nullptr;
                e.R = a.H[l + 1];
                e.RT = TRAIN ? a.HT[l + 1] : nullptr;
                tile_epilogue<kEpiHidden>(tmem, true, a.n, N, m0, n0, e, bias, colw, lossw, nullptr);
            } else if (i + 1 == L) {
                if constexpr (TRAIN) {
                    e.T = a.T;
                    e.vec = a.ovec;
                    e.R = L > 1 ? a.G[l] : nullptr;
                    e.RT = a.GT[l];
                    e.colpart = a.colpart[l];
                    e.losspart = a.losspart;
                    e.scale = a.scale;
                    tile_epilogue<kEpiLoss>(tmem, true, a.n, N, m0, n0, e, bias, colw, lossw, nullptr);
                } else {
                    e.Y = a.Y;
                    e.vec = a.ovec;
                    tile_epilogue<kEpiOut>(tmem, true, a.n, N, m0, n0, e, bias, colw, lossw, nullptr);
                }
            } else if constexpr (TRAIN) {
                e.Z = a.Z[l - 1];
                e.R = l > 1 ? a.G[l - 1] : nullptr;
                e.RT = a.GT[l - 1];
                e.colpart = a.colpart[l - 1];
                tile_epilogue<kEpiBack>(tmem, true, a.n, N, m0, n0, e, bias, colw, lossw, nullptr);
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (i + 1 < steps) cluster_barrier();   // the layer's columns of all four CTAs are in memory
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TC_TMEM_COLS) : "memory");
}

// What the kernels leave for the host, in page-locked memory mapped into the
// device's address space: read after the stream is synchronised, no copy.
struct alignas(64) HostSlot {
    double loss;
    int tc_err;   // set by a tensor-core wait that ran out
};

// Slots of all networks of the process, in page-locked slabs of 4 KiB: a
// cudaHostAlloc that has to map a new range costs 2.9 ms and its release 0.9
// (2.4 and 3.6 us out of one that is there), and a network is made in less.
// One slab stays for the next network, the others go with their last slot.
class HostSlots {
    static constexpr int kSlots = 64;
    struct Slab {
        HostSlot *mem;
        uint64_t used;
    };
    std::mutex lock;
    std::vector<Slab> slabs;

    // still page-locked memory (a cudaDeviceReset takes it away)?
    static bool alive(const HostSlot *mem)
    {
        cudaPointerAttributes at{};
        const bool ok = cudaPointerGetAttributes(&at, mem) == cudaSuccess && at.type == cudaMemoryTypeHost;
        cudaGetLastError();
        return ok;
    }

public:
    HostSlot *take()
    {
        std::lock_guard<std::mutex> hold(lock);
        for (size_t i = 0; i < slabs.size();) {
            if (!alive(slabs[i].mem)) {
                slabs.erase(slabs.begin() + i);
                continue;
            }
            for (int k = 0; k < kSlots; ++k)
                if (!(slabs[i].used >> k & 1)) {
                    slabs[i].used |= uint64_t(1) << k;
                    return slabs[i].mem + k;
                }
            ++i;
        }
        slabs.reserve(slabs.size() + 1);
        HostSlot *mem = nullptr;
        if (cudaHostAlloc(reinterpret_cast<void **>(&mem), sizeof(HostSlot) * kSlots,
                          cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        slabs.push_back({mem, 1});
        return mem;
    }
    void give(HostSlot *s)
    {
        std::lock_guard<std::mutex> hold(lock);
        for (size_t i = 0; i < slabs.size(); ++i) {
            if (s < slabs[i].mem || s >= slabs[i].mem + kSlots) continue;
            slabs[i].used &= ~(uint64_t(1) << (s - slabs[i].mem));
            if (!slabs[i].used && slabs.size() > 1) {
                cudaFreeHost(slabs[i].mem);
                slabs.erase(slabs.begin() + i);
            }
            return;
        }
    }
};
// never destroyed: a network may outlive the library's other statics
HostSlots &host_slots()
{
    static HostSlots *const all = new HostSlots;
    return *all;
}

}  // namespace

struct pfk_mlp {
    int device = 0, nl = 0, max_batch = 0;
    unsigned char *arena = nullptr;           // the device memory behind every pointer below
    std::vector<int> dims;
    std::vector<long long> w_off, b_off;      // offsets in the parameter vector
    long long nparam = 0;
    float *p = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;   // FP32 params, grads, Adam moments
    // BF16 weights as rows of din (p's order) and as rows of dout; they change
    // only together with p (set_params, train_step)
    __nv_bfloat16 *wb = nullptr, *wt = nullptr;
    std::vector<float *> Z;                   // pre-activations of the hidden layers [max_batch x d_l]
    std::vector<__nv_bfloat16 *> H, HT;       // layer inputs (H[0] = network input), rows and transposed
    std::vector<__nv_bfloat16 *> G, GT;       // BF16 dZ per layer, rows and transposed
    float *part = nullptr;                    // parts of the weight gradients
    float *colpart = nullptr;                 // column sums of dZ per row tile, all layers
    double *losspart = nullptr;
    HostSlot *slot = nullptr, *d_slot = nullptr;
    long long ldt = 0;                        // row stride of the transposed buffers (max_batch, rounded up to 8)
    long long step = 0;
    std::string err;
};

namespace {

pfk_status mlp_fail(pfk_mlp *m, const std::string &msg, pfk_status s)
{
    if (m) m->err = msg;
    g_mlp_error = msg;
    return s;
}

#define MLP_CK(call)                                                                            \
    do {                                                                                        \
        cudaError_t e_ = (call);                                                                \
        if (e_ != cudaSuccess) return mlp_fail(m, std::string(#call) + ": " + cudaGetErrorString(e_), PFK_ERR_CUDA); \
    } while (0)

int row_tiles(int n) { return (n + TC_M - 1) / TC_M; }

// Weight-gradient tiles of the network, and the splits of the batch for n
// rows: enough that tiles x splits give every SM a CTA, at least 4 rounds of
// K each, at most kMaxSplits parts.  Measured on 112-256-256-232 at 2048 rows
// (20 tiles): 8 splits.
constexpr int kMaxSplits = 16;

int weight_tiles(const std::vector<int> &d)
{
    int t = 0;
    for (size_t l = 0; l + 1 < d.size(); ++l) t += row_tiles(d[l]) * ((d[l + 1] + TC_N - 1) / TC_N);
    return t;
}

int split_cap(int tiles) { return std::max(1, std::min(kMaxSplits, 2 * 148 / tiles)); }

Layers layers_for(const pfk_mlp *m, int n)
{
    Layers L{};
    L.nl = m->nl;
    long long col = 0;
    int t = 0;
    for (int l = 0; l < m->nl; ++l) {
        L.din[l] = m->dims[l];
        L.dout[l] = m->dims[l + 1];
        L.tile0[l] = t;
        t += row_tiles(L.din[l]) * ((L.dout[l] + TC_N - 1) / TC_N);
        L.w_off[l] = m->w_off[l];
        L.b_off[l] = m->b_off[l];
        L.col_off[l] = col;
        col += (long long)row_tiles(m->max_batch) * L.dout[l];
        L.HT[l] = m->HT[l];
        L.GT[l] = m->GT[l];
    }
    L.tiles = t;
    const int rounds = (n + TC_K - 1) / TC_K;
    const int want = std::max(1, std::min(split_cap(t), rounds / 4));
    const int per = (rounds + want - 1) / want;
    L.ksplit = per * TC_K;
    L.splits = (rounds + per - 1) / per;
    return L;
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <int EPI>
void gemm(pfk_mlp *m, int M, int N, int K, const __nv_bfloat16 *A, const __nv_bfloat16 *B, const EpiArgs &e,
          cudaStream_t st)
{
    dim3 grid((N + TC_N - 1) / TC_N, row_tiles(M));
    launch_after(gemm_tc_kernel<EPI>, grid, TC_THREADS, TC_SMEM, st, M, N, K, A, B, e, &m->d_slot->tc_err);
}

bool fusable(const pfk_mlp *m)
{
    for (int d : m->dims)
        if (d > kFuseWidth) return false;
    return true;
}

// The fused kernel over n rows: forward to Y, or, with T, everything up to the
// weight gradients.
void fused(pfk_mlp *m, int n, const float *X, float *Y, const float *T, cudaStream_t st)
{
    FusedArgs a{};
    a.n = n;
    a.nl = m->nl;
    a.X = X;
    a.T = T;
    a.Y = Y;
    long long col = 0;
    for (int l = 0; l < m->nl; ++l) {
        a.wt[l] = m->wt + m->w_off[l];
        a.wb[l] = m->wb + m->w_off[l];
        a.bias[l] = m->p + m->b_off[l];
        a.Z[l] = m->Z[l];
        a.H[l] = m->H[l];
        a.HT[l] = m->HT[l];
        a.G[l] = m->G[l];
        a.GT[l] = m->GT[l];
        a.colpart[l] = m->colpart + col;
        col += (long long)row_tiles(m->max_batch) * m->dims[l + 1];
    }
    for (int l = 0; l <= m->nl; ++l) a.dims[l] = m->dims[l];
    a.losspart = m->losspart;
    a.ldt = m->ldt;
    a.scale = 1.0f / (float)((long long)n * m->dims[m->nl]);
    a.xvec = aligned16(X);
    a.ovec = aligned16(T ? (const void *)T : (const void *)Y);
    const dim3 grid(kFuseCtas, row_tiles(n));
    if (T) fused_kernel<true><<<grid, TC_THREADS, TC_SMEM, st>>>(a, &m->d_slot->tc_err);
    else fused_kernel<false><<<grid, TC_THREADS, TC_SMEM, st>>>(a, &m->d_slot->tc_err);
}

// Whether the n rows of Y share memory with the n rows of X.
bool overlaps(const pfk_mlp *m, int n, const float *X, const float *Y)
{
    const uintptr_t x = reinterpret_cast<uintptr_t>(X), y = reinterpret_cast<uintptr_t>(Y);
    return y < x + sizeof(float) * (size_t)n * m->dims[0] && x < y + sizeof(float) * (size_t)n * m->dims[m->nl];
}

// Forward pass of n rows of X: to Y, or, with T, to dZ of the last layer and the loss.
void forward(pfk_mlp *m, int n, const float *X, float *Y, const float *T, cudaStream_t st)
{
    // the fused kernel's clusters write their rows of Y while others still
    // read X; layer by layer, all of X is converted before Y is written
    if (fusable(m) && (T || !overlaps(m, n, X, Y))) return fused(m, n, X, Y, T, st);
    const bool train = T != nullptr;
    const int d0 = m->dims[0];
    dim3 gi((n + 31) / 32, (d0 + 31) / 32);
    input_kernel<<<gi, 256, 0, st>>>(X, n, d0, m->H[0], train ? m->HT[0] : nullptr, m->ldt);
    long long col = 0;
    for (int l = 0; l < m->nl; ++l) {
        const int din = m->dims[l], dout = m->dims[l + 1];
        EpiArgs e{};
        e.bias = m->p + m->b_off[l];
        e.ldt = m->ldt;
        const __nv_bfloat16 *w = m->wt + m->w_off[l];
        if (l + 1 < m->nl) {
            e.Z = train ? m->Z[l] : nullptr;
            e.R = m->H[l + 1];
            e.RT = train ? m->HT[l + 1] : nullptr;
            gemm<kEpiHidden>(m, n, dout, din, m->H[l], w, e, st);
        } else if (train) {
            e.T = T;
            e.vec = aligned16(T);
            e.R = m->nl > 1 ? m->G[l] : nullptr;
            e.RT = m->GT[l];
            e.colpart = m->colpart + col;
            e.losspart = m->losspart;
            e.scale = 1.0f / (float)((long long)n * dout);
            gemm<kEpiLoss>(m, n, dout, din, m->H[l], w, e, st);
        } else {
            e.Y = Y;
            e.vec = aligned16(Y);
            gemm<kEpiOut>(m, n, dout, din, m->H[l], w, e, st);
        }
        col += (long long)row_tiles(m->max_batch) * dout;
    }
}

// Gradient parts of the mean squared error after forward(..., T).
void backward(pfk_mlp *m, int n, const Layers &L, cudaStream_t st)
{
    for (int l = fusable(m) ? 0 : m->nl - 1; l > 0; --l) {
        // dH_{l-1} = G W_l^T (n x din); dZ_{l-1} = dH * SiLU'(Z_{l-1})
        EpiArgs e{};
        e.ldt = m->ldt;
        e.Z = m->Z[l - 1];
        e.R = l > 1 ? m->G[l - 1] : nullptr;
        e.RT = m->GT[l - 1];
        e.colpart = m->colpart + L.col_off[l - 1];
        gemm<kEpiBack>(m, n, m->dims[l], m->dims[l + 1], m->G[l], m->wb + m->w_off[l], e, st);
    }
    launch_after(gemm_dw_kernel, dim3(L.tiles, L.splits), TC_THREADS, TC_SMEM, st, L, n, m->ldt, m->part,
                 &m->d_slot->tc_err);
}

template <bool UPDATE>
void finish(pfk_mlp *m, int n, const Layers &L, const AdamArgs &a, cudaStream_t st)
{
    long long most = 0;
    for (int l = 0; l < m->nl; ++l) most = std::max(most, (long long)L.din[l] * L.dout[l] + L.dout[l]);
    const int nloss = row_tiles(n) * ((m->dims[m->nl] + TC_N - 1) / TC_N);
    launch_after(update_kernel<UPDATE>, dim3(blocks_for(most), m->nl), 256, 0, st, L, m->part, m->colpart,
                 row_tiles(n), m->losspart, nloss, &m->d_slot->loss, m->grad, m->p, m->m, m->v, m->wb, m->wt, a);
}

// After a synchronised call: PFK_ERR_CUDA if a GEMM's tensor-core wait ran out.
pfk_status check_tc(pfk_mlp *m)
{
    if (*(volatile int *)&m->slot->tc_err)
        return mlp_fail(m, "tensor-core GEMM: an mbarrier wait ran out (2 s)", PFK_ERR_CUDA);
    return PFK_OK;
}

pfk_status check_batch(pfk_mlp *m, const void *X, int n)
{
    if (!m) return mlp_fail(nullptr, "null network", PFK_ERR_STATE);
    if (!X || n <= 0 || n > m->max_batch) return mlp_fail(m, "null input or batch size outside 1..max_batch", PFK_ERR_INVALID);
    cudaSetDevice(m->device);
    return PFK_OK;
}

}  // namespace

extern "C" {

pfk_status pfk_mlp_create(int nlayers, const int *dims, int max_batch, int device, pfk_mlp **out)
{
    pfk_mlp *m = nullptr;
    if (!out) return mlp_fail(nullptr, "pfk_mlp_create: out is null", PFK_ERR_INVALID);
    *out = nullptr;
    if (nlayers < 1 || nlayers > 8 || !dims || max_batch <= 0)
        return mlp_fail(nullptr, "pfk_mlp_create: need 1..8 layers, dims and max_batch > 0", PFK_ERR_INVALID);
    for (int l = 0; l <= nlayers; ++l)
        if (dims[l] <= 0 || dims[l] > 4096 || dims[l] % 8)
            return mlp_fail(nullptr, "pfk_mlp_create: layer widths must be positive multiples of 8, at most 4096",
                            PFK_ERR_INVALID);
    m = new pfk_mlp();
    m->device = device;
    m->nl = nlayers;
    m->max_batch = max_batch;
    m->dims.assign(dims, dims + nlayers + 1);
    for (int l = 0; l < nlayers; ++l) {
        m->w_off.push_back(m->nparam);
        m->nparam += (long long)dims[l] * dims[l + 1];
        m->b_off.push_back(m->nparam);
        m->nparam += dims[l + 1];
    }
    auto bail = [&](pfk_status s) {
        g_mlp_error = m->err;
        pfk_mlp_destroy(m);
        return s;
    };
    if (cudaSetDevice(device) != cudaSuccess) return bail(mlp_fail(m, "cudaSetDevice failed", PFK_ERR_CUDA));
    // transposed buffers: rows of the batch rounded up to whole 16-byte segments
    m->ldt = ((long long)max_batch + 7) & ~7LL;
    const size_t rows = max_batch;
    const int tiles = weight_tiles(m->dims);
    long long cols = 0;
    for (int l = 0; l < nlayers; ++l) cols += (long long)row_tiles(max_batch) * dims[l + 1];
    const size_t nloss = (size_t)row_tiles(max_batch) * ((dims[nlayers] + TC_N - 1) / TC_N);
    for (auto *b : {&m->H, &m->HT, &m->G, &m->GT}) b->assign(nlayers, nullptr);
    m->Z.assign(nlayers, nullptr);
    // one allocation, carved in 256-byte steps: the first pass sizes it
    size_t total = 0;
    auto carve = [&]() {
        size_t at = 0;
        auto take = [&](auto *&q, size_t count) {
            if (m->arena) q = reinterpret_cast<std::remove_reference_t<decltype(q)>>(m->arena + at);
            at += (sizeof(*q) * count + 255) & ~size_t(255);
        };
        for (float **q : {&m->p, &m->m, &m->v, &m->grad}) take(*q, m->nparam);
        for (__nv_bfloat16 **q : {&m->wb, &m->wt}) take(*q, m->nparam);
        take(m->part, (size_t)tiles * split_cap(tiles) * TC_M * TC_N);
        take(m->colpart, cols);
        take(m->losspart, nloss);
        for (int l = 0; l < nlayers; ++l) {
            take(m->H[l], rows * dims[l]);
            take(m->HT[l], (size_t)m->ldt * dims[l]);
            take(m->G[l], rows * dims[l + 1]);
            take(m->GT[l], (size_t)m->ldt * dims[l + 1]);
            if (l + 1 < nlayers) take(m->Z[l], rows * dims[l + 1]);
        }
        total = at;
    };
    carve();
    bool ok = cudaMalloc(&m->arena, total) == cudaSuccess && (m->slot = host_slots().take()) &&
              cudaHostGetDevicePointer(reinterpret_cast<void **>(&m->d_slot), m->slot, 0) == cudaSuccess;
    if (ok) carve();
    if (!ok) return bail(mlp_fail(m, "pfk_mlp_create: device allocation failed", PFK_ERR_NOMEM));
    // the product kernels' shared-memory limits on this device
    for (const void *k : {(const void *)gemm_tc_kernel<kEpiHidden>, (const void *)gemm_tc_kernel<kEpiOut>,
                          (const void *)gemm_tc_kernel<kEpiLoss>, (const void *)gemm_tc_kernel<kEpiBack>,
                          (const void *)gemm_dw_kernel, (const void *)fused_kernel<true>,
                          (const void *)fused_kernel<false>})
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM) != cudaSuccess)
            return bail(mlp_fail(m, "pfk_mlp_create: kernel configuration failed", PFK_ERR_CUDA));
    m->slot->loss = 0.0;
    m->slot->tc_err = 0;
    cudaMemset(m->arena, 0, reinterpret_cast<unsigned char *>(m->part) - m->arena);   // parameters, moments, weights
    cudaStreamSynchronize(nullptr);
    *out = m;
    return PFK_OK;
}

pfk_status pfk_mlp_destroy(pfk_mlp *m)
{
    if (!m) return PFK_OK;
    cudaSetDevice(m->device);
    cudaDeviceSynchronize();
    if (m->arena) cudaFree(m->arena);
    if (m->slot) host_slots().give(m->slot);
    delete m;
    return PFK_OK;
}

const char *pfk_mlp_last_error(const pfk_mlp *m) { return m ? m->err.c_str() : g_mlp_error.c_str(); }

long long pfk_mlp_param_count(const pfk_mlp *m) { return m ? m->nparam : 0; }

pfk_status pfk_mlp_set_params(pfk_mlp *m, const float *params)
{
    if (!m || !params) return mlp_fail(m, "null network or parameters", PFK_ERR_INVALID);
    cudaSetDevice(m->device);
    MLP_CK(cudaMemcpy(m->p, params, sizeof(float) * m->nparam, cudaMemcpyHostToDevice));
    MLP_CK(cudaMemset(m->m, 0, sizeof(float) * m->nparam));
    MLP_CK(cudaMemset(m->v, 0, sizeof(float) * m->nparam));
    long long most = 0;
    for (int l = 0; l < m->nl; ++l) most = std::max(most, (long long)m->dims[l] * m->dims[l + 1]);
    weights_kernel<<<dim3(blocks_for(most), m->nl), 256>>>(m->p, layers_for(m, 1), m->wb, m->wt);
    MLP_CK(cudaGetLastError());
    MLP_CK(cudaStreamSynchronize(nullptr));   // the calls that use them may run on any stream
    m->step = 0;
    return PFK_OK;
}

pfk_status pfk_mlp_get_params(pfk_mlp *m, float *params)
{
    if (!m || !params) return mlp_fail(m, "null network or parameters", PFK_ERR_INVALID);
    cudaSetDevice(m->device);
    MLP_CK(cudaMemcpy(params, m->p, sizeof(float) * m->nparam, cudaMemcpyDeviceToHost));
    return PFK_OK;
}

pfk_status pfk_mlp_forward(pfk_mlp *m, const float *dX, int n, float *dY, void *stream)
{
    pfk_status s = check_batch(m, dX, n);
    if (s != PFK_OK) return s;
    if (!dY) return mlp_fail(m, "null output", PFK_ERR_INVALID);
    cudaStream_t st = (cudaStream_t)stream;
    forward(m, n, dX, dY, nullptr, st);
    MLP_CK(cudaGetLastError());
    MLP_CK(cudaStreamSynchronize(st));
    return check_tc(m);
}

pfk_status pfk_mlp_gradients(pfk_mlp *m, const float *dX, const float *dT, int n, float *grads, double *loss,
                             void *stream)
{
    pfk_status s = check_batch(m, dX, n);
    if (s != PFK_OK) return s;
    if (!dT) return mlp_fail(m, "null targets", PFK_ERR_INVALID);
    cudaStream_t st = (cudaStream_t)stream;
    const Layers L = layers_for(m, n);
    forward(m, n, dX, nullptr, dT, st);
    backward(m, n, L, st);
    finish<false>(m, n, L, AdamArgs{}, st);
    MLP_CK(cudaGetLastError());
    if (grads) MLP_CK(cudaMemcpyAsync(grads, m->grad, sizeof(float) * m->nparam, cudaMemcpyDeviceToHost, st));
    MLP_CK(cudaStreamSynchronize(st));
    if (loss) *loss = *(volatile double *)&m->slot->loss;
    return check_tc(m);
}

pfk_status pfk_mlp_train_step(pfk_mlp *m, const float *dX, const float *dT, int n, float lr, double *loss,
                              void *stream)
{
    pfk_status s = check_batch(m, dX, n);
    if (s != PFK_OK) return s;
    if (!dT || !(lr > 0.0f)) return mlp_fail(m, "null targets or non-positive learning rate", PFK_ERR_INVALID);
    cudaStream_t st = (cudaStream_t)stream;
    const Layers L = layers_for(m, n);
    forward(m, n, dX, nullptr, dT, st);
    backward(m, n, L, st);
    m->step += 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f / (1.0f - powf(b1, (float)m->step)), c2 = 1.0f / (1.0f - powf(b2, (float)m->step));
    finish<true>(m, n, L, AdamArgs{lr, b1, b2, 1e-8f, c1, c2}, st);
    MLP_CK(cudaGetLastError());
    MLP_CK(cudaStreamSynchronize(st));
    if (loss) *loss = *(volatile double *)&m->slot->loss;
    return check_tc(m);
}

}  // extern "C"

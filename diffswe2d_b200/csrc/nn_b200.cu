// nn_b200.cu -- training and inference kernels of the warm-start network.
//
// The matrix products run on the 5th-generation tensor cores: one CTA of
// nine warps computes a 128 x bn tile of A B^T (bf16 operands, fp32
// accumulator in tensor memory).  Eight warps stage the operands global ->
// shared memory by cp.async in the 128-byte-swizzled K-major layout that
// tcgen05.mma reads through shared-memory matrix descriptors, up to eight
// stages deep; one thread of the ninth issues the MMAs and commits them to
// the stage's mbarrier; the epilogue reads the accumulator with tcgen05.ld
// (each warp its 32 lanes) and applies bias and activation.  Every mbarrier
// wait is bounded in time: a wait inside the K loop gives up after the
// launch's limit (wait_ns), after which the CTA records error bit 1, stops
// issuing, waits for its issued MMAs to drain (a fixed, separate bound of
// 2 s), frees its tensor memory and returns.  If the drain bound also runs
// out, the CTA still frees its tensor memory (every allocation must be freed
// before the CTA exits) and records error bit 2: MMAs may then have been
// running when it was freed, and the context should not be trusted.
//
// The rest are small memory-bound kernels (im2col / col2im for the 1D
// convolutions, activation adjoint, transposes, column sums, MSE, Adam).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/nn_b200.h"
#include "../../include/swe_b200.h"

namespace nn {
namespace {

constexpr int BM = 128;       // tile rows (UMMA M)
constexpr int BK = 64;        // K elements per stage
constexpr int BN_MAX = 128;   // tile columns (UMMA N): 16, 32, 64 or 128
constexpr int LOADERS = 8;    // warps that stage operands
constexpr int NT = 32 * (LOADERS + 1);
constexpr int STAGES_MAX = 8;
// A K-major operand tile: one 128-byte row (64 bf16) per matrix row, its
// sixteen-byte chunk c stored at position c ^ (row & 7) (the 128-byte
// swizzle; the tile starts on a 1,024-byte boundary).
__host__ __device__ constexpr int tile_bytes(int rows) { return rows * BK * 2; }
// Bound of the final wait for the CTA's own MMAs before its tensor memory is
// freed (independent of the launch's wait limit, so that a short limit
// never frees tensor memory under MMAs that are still running).
constexpr unsigned long long DRAIN_LIMIT_NS = 2000000000ull;  // 2 s

// Dynamic shared memory of a launch: up to eight stages of the narrower
// tiles, four of the widest.
constexpr int SMEM_ALIGN = 1024;
constexpr int SMEM_MAX = STAGES_MAX * (tile_bytes(BM) + tile_bytes(64));
static_assert(SMEM_MAX + SMEM_ALIGN + 1024 <= 227 * 1024 && 4 * (tile_bytes(BM) + tile_bytes(BN_MAX)) <= SMEM_MAX, "");

struct GemmArgs {
    const uint16_t* A;
    const uint16_t* B;
    int M, N, K, lda, ldb, kchunk;  // kchunk: K per blockIdx.z (multiple of BK)
    int bn, stages;                 // tile columns, pipeline stages
    const float* bias;
    int act, ldc;
    float* out_f32;
    uint16_t* out_bf16;
    float* pre_f32;
    float* partial;  // split K: [z][M][N]
    uint32_t* err;
    unsigned long long wait_ns;  // limit of each wait inside the K loop
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Shared-memory matrix descriptor of a K-major tile in the 128-byte swizzle:
// 1,024 bytes between 8-row groups (bits 32-45; the leading offset, bits
// 16-29, is not used by this layout), version 1 (bits 46-47), layout 2
// (bits 61-63).  A K step of 16 elements is 32 bytes further on.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) |
           (2ull << 61);
}

// Instruction descriptor of kind::f16: fp32 accumulator (bits 4-5 = 1),
// A and B bf16 (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bit 17,
// M >> 4 at bit 24.
__device__ __forceinline__ uint32_t instr_desc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(BM >> 4) << 24);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.shared::cta.b64 t, [%0];\n\t}" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Wait for the phase `parity` of an mbarrier, giving up once `limit`
// nanoseconds have passed (a limit of 0 gives up at once).  The clock is
// read only after a first run of probes: a read of globaltimer costs more
// than a K block (0.9 us a block with the clock read before every probe).
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, unsigned long long limit) {
    for (int i = 0; i < 256; ++i)
        if (mbar_try(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    while (global_ns() - t0 < limit) {
        if (mbar_try(bar, parity)) return true;
    }
    return false;
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, unsigned long long limit) {
    if (limit == 0) return false;
    return mbar_try(bar, parity) || mbar_wait_slow(bar, parity, limit);
}

// One lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                         uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
        "[%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 16 bytes global -> shared, zero-filled where !ok (src is then not read).
__device__ __forceinline__ void cp16(uint32_t dst, const uint16_t* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0)
                 : "memory");
}

__device__ __forceinline__ float gelu(float x) {
    return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f));
}

__device__ __forceinline__ float gelu_grad(float x) {
    // d/dx x Phi(x) = Phi(x) + x phi(x)
    const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
    return cdf + x * pdf;
}

__device__ __forceinline__ void epilogue_store(const GemmArgs& g, int r, int c, float acc) {
    float pre = acc + (g.bias ? g.bias[c] : 0.0f);
    const float y = g.act == NN_ACT_GELU ? gelu(pre) : pre;
    const size_t o = (size_t)r * g.ldc + c;
    if (g.pre_f32) g.pre_f32[o] = pre;
    if (g.out_f32) g.out_f32[o] = y;
    if (g.out_bf16) g.out_bf16[o] = __bfloat16_as_ushort(__float2bfloat16_rn(y));
}

// Whether four values at o, o + 1, ... of p can be written by one 16-byte
// store (o a multiple of 4 with ldc, checked here with the base's alignment).
__device__ __forceinline__ bool vec4_ok(const void* p, int ldc, int bytes) {
    return (((uintptr_t)p & (uintptr_t)(4 * bytes - 1)) | (uintptr_t)(ldc & 3)) == 0;
}

// 16 consecutive accumulators of row r from column c on.
__device__ __forceinline__ void epilogue16(const GemmArgs& g, int r, int c, const float (&v)[16], bool vec) {
    if (g.partial) {
        float* p = g.partial + ((size_t)blockIdx.z * g.M + r) * g.N + c;
        if (vec && c + 16 <= g.N) {
#pragma unroll
            for (int i = 0; i < 16; i += 4)
                *reinterpret_cast<float4*>(p + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (c + i < g.N) p[i] = v[i];
        }
        return;
    }
    if (!vec || c + 16 > g.N) {
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (c + i < g.N) epilogue_store(g, r, c + i, v[i]);
        return;
    }
    const size_t o = (size_t)r * g.ldc + c;
#pragma unroll
    for (int i = 0; i < 16; i += 4) {
        float pre[4], y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            pre[e] = v[i + e] + (g.bias ? g.bias[c + i + e] : 0.0f);
            y[e] = g.act == NN_ACT_GELU ? gelu(pre[e]) : pre[e];
        }
        if (g.pre_f32) *reinterpret_cast<float4*>(g.pre_f32 + o + i) = make_float4(pre[0], pre[1], pre[2], pre[3]);
        if (g.out_f32) *reinterpret_cast<float4*>(g.out_f32 + o + i) = make_float4(y[0], y[1], y[2], y[3]);
        if (g.out_bf16) {
            ushort4 b;
            b.x = __bfloat16_as_ushort(__float2bfloat16_rn(y[0]));
            b.y = __bfloat16_as_ushort(__float2bfloat16_rn(y[1]));
            b.z = __bfloat16_as_ushort(__float2bfloat16_rn(y[2]));
            b.w = __bfloat16_as_ushort(__float2bfloat16_rn(y[3]));
            *reinterpret_cast<ushort4*>(g.out_bf16 + o + i) = b;
        }
    }
}

// Stage columns [k0, k0 + BK) of `rows` rows from row0 on (rows at or past
// `limit` and columns at or past kend read as zero), the share of part `part`
// of `parts` warps: eight lanes per row, one 16-byte chunk each.  A row stays
// within 128 bytes of shared memory: with the chunks of a row spread over the
// tile (the unswizzled layout) each 32-byte sector that arrives is split
// (17,920 x 64 x 384: 22.5 us against 16.5 at otherwise the same code).
__device__ __forceinline__ void stage_tile(uint32_t smem, const uint16_t* base, int ld, int row0, int limit,
                                           int rows, int k0, int kend, int part, int parts) {
    const int lane = threadIdx.x & 31, kc = lane & 7;
    const int k = k0 + kc * 8;
    const bool kin = k < kend;
    const int r0 = part * 4 + (lane >> 3);
    const uint16_t* src = base + (size_t)(row0 + r0) * ld + k;
    const size_t step = (size_t)(4 * parts) * ld;
    const int left = limit - row0;
#pragma unroll 4
    for (int r = r0; r < rows; r += 4 * parts, src += step) {
        const bool ok = kin && r < left;
        cp16(smem + r * 128 + ((kc ^ (r & 7)) << 4), ok ? src : base, ok);
    }
}

// The network's products are small (a CTA walks up to 70 K blocks of 18 to
// 33 KB), so what bounds this kernel is how many blocks' loads are in flight.
// Each loader warp has a stage of its own (two or more share one where K is
// short): it copies the stage, waits for the copies, makes them visible to
// the tensor core and only then goes on, so that the eight stages' latencies
// overlap without one warp's proxy fence waiting for another's copies.  The
// tile is narrowed until the grid fills the chip.  The K order of every
// element's sum does not depend on any of this, so neither do its bits.
// Measured against 128 threads that load a stage, issue its MMAs and only
// then load the next: 256 x 96 x 4480 226 -> 20 us, the 17 products of a
// training step of 256 runs 764 -> 160 us.
__global__ void __launch_bounds__(NT, 1) gemm_kernel(const GemmArgs g) {
    extern __shared__ uint8_t smem[];
    __shared__ uint64_t s_full[STAGES_MAX], s_free[STAGES_MAX];
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_ok;
    __shared__ int s_drained;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * BM;
    const int bn = g.bn, S = g.stages;
    const int n0 = blockIdx.y * bn;
    const int kbeg = blockIdx.z * g.kchunk;
    const int kend = min(g.K, kbeg + g.kchunk);
    const int nkb = kend > kbeg ? (kend - kbeg + BK - 1) / BK : 0;
    uint32_t ncols = 32;
    while ((int)ncols < bn) ncols <<= 1;

    const int parts = LOADERS / S;  // loader warps per stage (S is a power of two)
    if (warp == LOADERS) {          // tensor memory for the accumulator (one full warp)
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&s_tmem)), "r"(ncols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int i = 0; i < S; ++i) {
            mbar_init(smem_u32(&s_full[i]), (uint32_t)parts);
            mbar_init(smem_u32(&s_free[i]), 1u);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_ok = 1;
        s_drained = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    const uint32_t base = (smem_u32(smem) + 1023u) & ~1023u;
    const int stage_bytes = tile_bytes(BM) + tile_bytes(bn);
    const uint32_t full0 = smem_u32(&s_full[0]), free0 = smem_u32(&s_free[0]);
    const int log_s = 31 - __clz(S);

    // Stage kb % S holds block kb; its loads complete phase kb / S of the
    // stage's "full" barrier, its MMAs phase kb / S of its "free" barrier.
    if (warp < LOADERS) {
        const int st = warp / parts, part = warp - st * parts;
        const uint32_t sA = base + st * stage_bytes, sB = sA + tile_bytes(BM);
        const uint32_t full = full0 + 8 * st, freed = free0 + 8 * st;
        for (int kb = st; kb < nkb; kb += S) {
            if (kb >= S && !mbar_wait(freed, (uint32_t)(((kb >> log_s) - 1) & 1), g.wait_ns)) {
                s_ok = 0;
                break;
            }
            if (!s_ok) break;
            const int k0 = kbeg + kb * BK;
            stage_tile(sA, g.A, g.lda, m0, g.M, BM, k0, kend, part, parts);
            stage_tile(sB, g.B, g.ldb, n0, g.N, bn, k0, kend, part, parts);
            asm volatile("cp.async.wait_all;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(full);
        }
    } else {
        // The whole warp walks the K loop (uniform control flow and operands;
        // one thread in a divergent branch took 1,150 cycles a block, twice
        // the loads' share) and one elected lane issues.
        const uint32_t idesc = instr_desc(bn);
        const uint64_t descA = smem_desc(base), descB = smem_desc(base + tile_bytes(BM));
        const uint32_t stage_step = (uint32_t)stage_bytes >> 4;  // in descriptor address units
        const bool issuer = elect_one();
        const int ktail = (kend - kbeg) - (nkb - 1) * BK;  // columns of the last block
        bool good = true;
        int kb = 0;
        for (; kb < nkb; ++kb) {
            const int st = kb & (S - 1);
            // the first two blocks' waits are for loads alone
            good = mbar_wait(full0 + 8 * st, (uint32_t)((kb >> log_s) & 1), kb < 2 ? DRAIN_LIMIT_NS : g.wait_ns);
            if (!__all_sync(0xffffffffu, good)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t ad = descA + st * stage_step, bd = descB + st * stage_step;
            if (issuer) {
                if (kb + 1 < nkb || ktail == BK) {
#pragma unroll
                    for (int t = 0; t < BK / 16; ++t)
                        mma_bf16(tmem, ad + 2 * t, bd + 2 * t, idesc, (kb > 0 || t > 0) ? 1u : 0u);
                } else {
                    for (int t = 0; t * 16 < ktail; ++t)
                        mma_bf16(tmem, ad + 2 * t, bd + 2 * t, idesc, (kb > 0 || t > 0) ? 1u : 0u);
                }
                mma_commit(free0 + 8 * st);
            }
            __syncwarp();
        }
        if (kb < nkb) s_ok = 0;
        // Wait for the last commit (it covers every MMA issued).
        if (kb > 0) {
            const int last = kb - 1;
            if (!mbar_wait(free0 + 8 * (last & (S - 1)), (uint32_t)((last >> log_s) & 1), DRAIN_LIMIT_NS))
                s_drained = 0;
        }
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const bool ok = s_ok != 0 && s_drained != 0;
    if (!ok) {
        if (tid == 0 && g.err) atomicOr(g.err, (s_ok ? 0u : 1u) | (s_drained ? 0u : 2u));
    } else if (warp < LOADERS) {
        // warps w and w + 4 share the rows of TMEM lanes 32 (w % 4) ..
        const int r = m0 + (warp & 3) * 32 + lane;
        const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const bool vec = g.partial ? vec4_ok(g.partial, g.N, 4)
                                   : vec4_ok(g.out_f32, g.ldc, 4) && vec4_ok(g.pre_f32, g.ldc, 4) &&
                                         vec4_ok(g.out_bf16, g.ldc, 2);
        for (int c0 = (warp >> 2) * 16; c0 < bn && n0 + c0 < g.N; c0 += 32) {
            float v[16];
            if (nkb > 0) {
                tmem_ld16(lane_addr + (uint32_t)c0, v);
            } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = 0.0f;
            }
            if (r < g.M) epilogue16(g, r, n0 + c0, v, vec);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == LOADERS)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols));
}

// Split-K: sum the partial tiles in z order, then the epilogue.
__global__ void splitk_epilogue_kernel(const GemmArgs g, int ksplit) {
    const long long total = (long long)g.M * g.N;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        float acc = 0.0f;
        for (int z = 0; z < ksplit; ++z) acc += g.partial[(size_t)z * total + i];
        const int r = (int)(i / g.N), c = (int)(i - (long long)r * g.N);
        epilogue_store(g, r, c, acc);
    }
}

__device__ __forceinline__ float bf16_to_f(uint16_t u) { return __uint_as_float((uint32_t)u << 16); }
__device__ __forceinline__ uint16_t f_to_bf16(float f) {
    return __bfloat16_as_ushort(__float2bfloat16_rn(f));
}

__global__ void im2col_kernel(const float* xf, const uint16_t* xb, int Nb, int Lin, int Cin, int sn,
                              int sl, int sc, int k, int stride, int pad, int Lout, float scale,
                              float shift, uint16_t* cols, int ldcols) {
    const long long total = (long long)Nb * Lout * ldcols;
    const int kc = k * Cin;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long row = i / ldcols;
        const int col = (int)(i - row * ldcols);
        float v = 0.0f;
        if (col < kc) {
            const int n = (int)(row / Lout), lo = (int)(row - (long long)n * Lout);
            const int kk = col / Cin, ci = col - kk * Cin;
            const int l = lo * stride - pad + kk;
            if (l >= 0 && l < Lin) {
                const size_t o = (size_t)n * sn + (size_t)l * sl + (size_t)ci * sc;
                v = (xf ? xf[o] : bf16_to_f(xb[o])) * scale + shift;
            }
        }
        cols[i] = f_to_bf16(v);
    }
}

__global__ void col2im_kernel(const float* dcols, int ld, int Nb, int Lin, int Cin, int k, int stride,
                              int pad, int Lout, float* dX) {
    const long long total = (long long)Nb * Lin * Cin;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int ci = (int)(i % Cin);
        const long long nl = i / Cin;
        const int l = (int)(nl % Lin), n = (int)(nl / Lin);
        float acc = 0.0f;
        // kk = l + pad - lo*stride in [0, k)
        for (int kk = (l + pad) % stride; kk < k; kk += stride) {
            const int lo = (l + pad - kk) / stride;
            if (lo < 0 || lo >= Lout) continue;
            acc += dcols[((size_t)n * Lout + lo) * ld + (size_t)kk * Cin + ci];
        }
        dX[i] = acc;
    }
}

__global__ void act_backward_kernel(const float* dact, const float* pre, int M, int N, int ld_in,
                                    int act, uint16_t* d_bf16, int ldd, uint16_t* dT_bf16, int ldt,
                                    float* d_f32) {
    // 32 x 32 tiles through shared memory so the transposed store is coalesced.
    __shared__ uint16_t tile[32][33];
    const int bx = blockIdx.x * 32, by = blockIdx.y * 32;  // bx: column (N), by: row (M)
    const int tx = threadIdx.x, ty = threadIdx.y;           // 32 x 8 threads
    for (int j = ty; j < 32; j += 8) {
        const int r = by + j, c = bx + tx;
        uint16_t b = 0;
        if (r < M && c < N) {
            const size_t o = (size_t)r * ld_in + c;
            float d = dact[o];
            if (act == NN_ACT_GELU) d *= gelu_grad(pre[o]);
            b = f_to_bf16(d);
            if (d_bf16) d_bf16[(size_t)r * ldd + c] = b;
            if (d_f32) d_f32[(size_t)r * ld_in + c] = d;
        }
        tile[j][tx] = b;
    }
    __syncthreads();
    if (!dT_bf16) return;
    for (int j = ty; j < 32; j += 8) {
        const int c = bx + j, r = by + tx;  // write dT[c][r]
        if (c < N && r < ldt) dT_bf16[(size_t)c * ldt + r] = r < M ? tile[tx][j] : (uint16_t)0;
    }
}

__global__ void colsum_kernel(const float* x, int M, int N, int ld, float* out) {
    const int c = blockIdx.x;
    __shared__ float s[256];
    float acc = 0.0f;
    for (int r = threadIdx.x; r < M; r += blockDim.x) acc += x[(size_t)r * ld + c];
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[c] = s[0];
}

__global__ void transpose_bf16_kernel(const uint16_t* in, int R, int C, int ldi, uint16_t* out,
                                      int ldo) {
    __shared__ uint16_t tile[32][33];
    const int bc = blockIdx.x * 32, br = blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int j = ty; j < 32; j += 8) {
        const int r = br + j, c = bc + tx;
        tile[j][tx] = (r < R && c < C) ? in[(size_t)r * ldi + c] : (uint16_t)0;
    }
    __syncthreads();
    for (int j = ty; j < 32; j += 8) {
        const int c = bc + j, r = br + tx;
        if (c < C && r < ldo) out[(size_t)c * ldo + r] = r < R ? tile[tx][j] : (uint16_t)0;
    }
}

__global__ void cast_kernel(const float* in, int R, int C, int ldi, uint16_t* out, int ldo) {
    const long long total = (long long)R * ldo;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long r = i / ldo;
        const int c = (int)(i - r * ldo);
        out[i] = c < C ? f_to_bf16(in[(size_t)r * ldi + c]) : (uint16_t)0;
    }
}

__global__ void mse_kernel(const float* pred, const float* target, int M, int N, float* loss,
                           float* grad) {
    __shared__ float s[256];
    const long long total = (long long)M * N;
    const float inv = 1.0f / (float)total;
    float acc = 0.0f;
    for (long long i = threadIdx.x; i < total; i += blockDim.x) {
        const float d = pred[i] - target[i];
        acc += d * d;
        if (grad) grad[i] = 2.0f * d * inv;
    }
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0 && loss) loss[0] = s[0] * inv;
}

__global__ void adam_kernel(float* p, const float* g, float* m, float* v, long long count, float lr,
                            float b1, float b2, float eps, float c1, float c2) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count;
         i += (long long)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

int grid_for(long long n, int threads) {
    long long b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    return (int)(b > 148LL * 16 ? 148LL * 16 : b);
}

bool g_smem_set[64] = {false};

}  // namespace
}  // namespace nn

using namespace nn;

extern "C" int nn_gemm_bf16(const uint16_t* A, int lda, const uint16_t* B, int ldb, int M, int N,
                            int K, const float* bias, int act, float* out_f32, uint16_t* out_bf16,
                            float* pre_f32, int ldc, int ksplit, float* workspace,
                            long long wait_ns, uint32_t* err, void* stream) {
    if (!A || !B || M < 1 || N < 1 || K < 16 || K % 16 || lda % 8 || ldb % 8 || lda < K || ldb < K)
        return SWE_EARG;
    if (wait_ns < 0) return SWE_EARG;
    if (((uintptr_t)A | (uintptr_t)B) & 15u) return SWE_EARG;
    if (act != NN_ACT_NONE && act != NN_ACT_GELU) return SWE_EARG;
    if (!out_f32 && !out_bf16 && !pre_f32) return SWE_EARG;
    if (ldc < N || ksplit < 1 || ksplit > 1024 || (ksplit > 1 && !workspace)) return SWE_EARG;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return SWE_ECUDA;
    if (!g_smem_set[dev]) {
        if (cudaFuncSetAttribute(gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 SMEM_MAX + SMEM_ALIGN) != cudaSuccess)
            return SWE_ECUDA;
        g_smem_set[dev] = true;
    }
    GemmArgs g{};
    g.A = A;
    g.B = B;
    g.M = M;
    g.N = N;
    g.K = K;
    g.lda = lda;
    g.ldb = ldb;
    // K per split, a multiple of BK
    const int kblocks = (K + BK - 1) / BK;
    const int per = (kblocks + ksplit - 1) / ksplit;
    g.kchunk = per * BK;
    const int zs = (kblocks + per - 1) / per;
    g.bias = bias;
    g.act = act;
    g.ldc = ldc;
    g.out_f32 = out_f32;
    g.out_bf16 = out_bf16;
    g.pre_f32 = pre_f32;
    g.partial = zs > 1 ? workspace : nullptr;
    g.err = err;
    g.wait_ns = (unsigned long long)wait_ns;
    cudaStream_t s = (cudaStream_t)stream;
    // Tile columns: the widest tile (A is read once per column tile) whose
    // grid still has a CTA for each SM, or the narrowest.
    int bn = BN_MAX;
    const long long mz = (long long)((M + BM - 1) / BM) * zs;
    while (bn > 16 && (bn / 2 >= N || mz * ((N + bn - 1) / bn) < 148)) bn /= 2;
    g.bn = bn;
    g.stages = 1;  // a power of two, no more than the K blocks need
    while (g.stages < per && g.stages < (bn == BN_MAX ? 4 : STAGES_MAX)) g.stages *= 2;
    const dim3 grid((M + BM - 1) / BM, (N + bn - 1) / bn, zs);
    gemm_kernel<<<grid, NT, g.stages * (tile_bytes(BM) + tile_bytes(bn)) + SMEM_ALIGN, s>>>(g);
    if (zs > 1) splitk_epilogue_kernel<<<grid_for((long long)M * N, 256), 256, 0, s>>>(g, zs);
    return cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

extern "C" int nn_im2col(const float* x_f32, const uint16_t* x_bf16, int Nb, int Lin, int Cin,
                         int x_stride_n, int x_stride_l, int x_stride_c, int k, int stride, int pad,
                         int Lout, float scale, float shift, uint16_t* cols, int ldcols,
                         void* stream) {
    if ((!x_f32 && !x_bf16) || !cols || Nb < 1 || Lin < 1 || Cin < 1 || k < 1 || stride < 1 ||
        pad < 0 || Lout < 1 || ldcols < k * Cin)
        return SWE_EARG;
    const long long total = (long long)Nb * Lout * ldcols;
    im2col_kernel<<<grid_for(total, 256), 256, 0, (cudaStream_t)stream>>>(
        x_f32, x_bf16, Nb, Lin, Cin, x_stride_n, x_stride_l, x_stride_c, k, stride, pad, Lout, scale,
        shift, cols, ldcols);
    return cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

extern "C" int nn_col2im(const float* dcols, int lddcols, int Nb, int Lin, int Cin, int k, int stride,
                         int pad, int Lout, float* dX, void* stream) {
    if (!dcols || !dX || Nb < 1 || Lin < 1 || Cin < 1 || k < 1 || stride < 1 || pad < 0 || Lout < 1 ||
        lddcols < k * Cin)
        return SWE_EARG;
    const long long total = (long long)Nb * Lin * Cin;
    col2im_kernel<<<grid_for(total, 256), 256, 0, (cudaStream_t)stream>>>(dcols, lddcols, Nb, Lin, Cin,
                                                                        k, stride, pad, Lout, dX);
    return cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

extern "C" int nn_act_backward(const float* dact, const float* pre, int M, int N, int ld_in, int act,
                               uint16_t* d_bf16, int ldd, uint16_t* dT_bf16, int ldt, float* d_f32,
                               void* stream) {
    if (!dact || M < 1 || N < 1 || ld_in < N || (act == NN_ACT_GELU && !pre)) return SWE_EARG;
    if (act != NN_ACT_NONE && act != NN_ACT_GELU) return SWE_EARG;
    if ((d_bf16 && ldd < N) || (dT_bf16 && ldt < M)) return SWE_EARG;
    const int Mt = dT_bf16 ? (ldt > M ? ldt : M) : M;  // rows covered (zero tail of dT)
    const dim3 grid((N + 31) / 32, (Mt + 31) / 32);
    act_backward_kernel<<<grid, dim3(32, 8), 0, (cudaStream_t)stream>>>(dact, pre, M, N, ld_in, act,
                                                                       d_bf16, ldd, dT_bf16, ldt, d_f32);
    return cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

extern "C" int nn_colsum(const float* x, int M, int N, int ld, float* out, void* stream) {
    if (!x || !out || M < 1 || N < 1 || ld < N) return SWE_EARG;
    colsum_kernel<<<N, 256, 0, (cudaStream_t)stream>>>(x, M, N, ld, out);
    return cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

extern "C" int nn_transpose_bf16(const uint16_t* in, int R, int C, int ldi, uint16_t* out, int ldo,
                                 void* stream) {
    if (!in || !out || R < 1 || C < 1 || ldi < C || ldo < R) return SWE_EARG;
    const dim3 grid((C + 31) / 32, (ldo + 31) / 32);
    transpose_bf16_kernel<<<grid, dim3(32, 8), 0, (cudaStream_t)stream>>>(in, R, C, ldi, out, ldo);
    return cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

extern "C" int nn_cast_bf16(const float* in, int R, int C, int ldi, uint16_t* out, int ldo,
                            uint16_t* outT, int ldt, void* stream) {
    if (!in || !out || R < 1 || C < 1 || ldi < C || ldo < C || (outT && ldt < R)) return SWE_EARG;
    cudaStream_t s = (cudaStream_t)stream;
    cast_kernel<<<grid_for((long long)R * ldo, 256), 256, 0, s>>>(in, R, C, ldi, out, ldo);
    if (outT) {
        const dim3 grid((C + 31) / 32, (ldt + 31) / 32);
        transpose_bf16_kernel<<<grid, dim3(32, 8), 0, s>>>(out, R, C, ldo, outT, ldt);
    }
    return cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

extern "C" int nn_mse(const float* pred, const float* target, int M, int N, float* loss, float* grad,
                      void* stream) {
    if (!pred || !target || M < 1 || N < 1) return SWE_EARG;
    mse_kernel<<<1, 256, 0, (cudaStream_t)stream>>>(pred, target, M, N, loss, grad);
    return cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

extern "C" int nn_adam(float* params, const float* grads, float* m, float* v, long long count, float lr,
                       float beta1, float beta2, float eps, int step, void* stream) {
    if (!params || !grads || !m || !v || count < 1 || step < 1) return SWE_EARG;
    const float c1 = 1.0f - powf(beta1, (float)step);
    const float c2 = 1.0f - powf(beta2, (float)step);
    adam_kernel<<<grid_for(count, 256), 256, 0, (cudaStream_t)stream>>>(params, grads, m, v, count, lr,
                                                                        beta1, beta2, eps, c1, c2);
    return cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

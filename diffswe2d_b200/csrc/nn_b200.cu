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

#include <algorithm>
#include <atomic>

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
// Operand tiles are stored in lines of 128 bytes (64 bf16), the sixteen-byte
// chunk c of line i at position c ^ (i & 7) (the 128-byte swizzle; a tile
// starts on a 1,024-byte boundary).  K-major: a line per row of the tile, BK
// elements of K.  MN-major: blocks of 64 rows, each BK lines (one per K).
__host__ __device__ constexpr int tile_bytes(int rows) { return rows * BK * 2; }
__host__ __device__ constexpr int mn_tile_bytes(int rows) { return (rows < 64 ? 64 : rows) * BK * 2; }
// Bound of the final wait for the CTA's own MMAs before its tensor memory is
// freed (independent of the launch's wait limit, so that a short limit
// never frees tensor memory under MMAs that are still running).
constexpr unsigned long long DRAIN_LIMIT_NS = 2000000000ull;  // 2 s

// Dynamic shared memory of a launch: up to eight stages of the narrower
// tiles, four of the widest.
constexpr int SMEM_ALIGN = 1024;
constexpr int SMEM_MAX = STAGES_MAX * (tile_bytes(BM) + tile_bytes(64));
// At least a quarter of an SM's shared memory (228 KB), so that no more than
// three CTAs of a launch share an SM whatever their registers allow: their
// allocations (at most 128 of its 512 tensor-memory columns each) never wait.
constexpr int SMEM_MIN = 57 * 1024;
static_assert(4 * SMEM_MIN >= 228 * 1024 && 3 * BN_MAX <= 512, "");
static_assert(SMEM_MAX + SMEM_ALIGN + 1024 <= 227 * 1024 && 4 * (tile_bytes(BM) + tile_bytes(BN_MAX)) <= SMEM_MAX, "");

// A GEMM operand in memory: lines of `cols` contiguous elements.  K-major: a
// line is a row of the product's operand (M or N index), its elements run
// along K.  MN-major: a line is one K index, its elements run along M or N.
// With lout > 0 the lines are the patches of a 1-D convolution read in place
// (line n * lout + l is elements [off + l * ld, ...) of sample n, whose
// `batch` elements are followed by the next sample's; elements outside the
// sample are zero padding).
struct Operand {
    const uint16_t* p;
    int ld, lines, cols;
    int lout, batch, off;
};

struct GemmArgs {
    Operand A, B;
    int M, N, K, kchunk;  // kchunk: K per blockIdx.z (multiple of BK)
    int bn, stages;       // tile columns, pipeline stages
    const float* bias;
    int act, ldc;
    float* out_f32;
    uint16_t* out_bf16;
    float* pre_f32;
    const float* adj_pre;  // activation adjoint: acc *= gelu'(adj_pre[r, c]) (ldc)
    float* colpart;        // then: column sums of each row tile [gridDim.x][N]
    float* partial;        // split K: [z][M][N]
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

// Shared-memory matrix descriptor in the 128-byte swizzle: address, leading
// offset (bits 16-29: MN-major, bytes between two blocks of 64 rows; not
// used K-major), stride offset (bits 32-45: 1,024 bytes between groups of
// eight lines), version 1 (bits 46-47), layout 2 (bits 61-63).  A K step of
// 16 elements is 32 bytes further on K-major, 16 lines MN-major.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, bool mn) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(mn ? (64 * BK * 2) >> 4 : 1) << 16) |
           ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
template <bool MN>
__host__ __device__ constexpr uint32_t k_step() { return MN ? (16 * 128) >> 4 : 32 >> 4; }

// Instruction descriptor of kind::f16: fp32 accumulator (bits 4-5 = 1),
// A and B bf16 (bits 7-9, 10-12 = 1), A / B MN-major (bits 15, 16),
// N >> 3 at bit 17, M >> 4 at bit 24.
__device__ __forceinline__ uint32_t instr_desc(int n, bool a_mn, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
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

// Sums over the warp's lanes of 16 values per lane: lane l returns the sum of
// value l >> 1 (a fixed order: halves exchanged at distances 16, 8, 4, 2, 1).
__device__ __forceinline__ float column_sum16(const float (&v)[16]) {
    const int lane = threadIdx.x & 31;
    float a[8], b[4], c[2], d;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const bool up = (lane & 16) != 0;
        const float keep = up ? v[i + 8] : v[i], give = up ? v[i] : v[i + 8];
        a[i] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const bool up = (lane & 8) != 0;
        const float keep = up ? a[i + 4] : a[i], give = up ? a[i] : a[i + 4];
        b[i] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const bool up = (lane & 4) != 0;
        const float keep = up ? b[i + 2] : b[i], give = up ? b[i] : b[i + 2];
        c[i] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
    }
    {
        const bool up = (lane & 2) != 0;
        const float keep = up ? c[1] : c[0], give = up ? c[0] : c[1];
        d = keep + __shfl_xor_sync(0xffffffffu, give, 2);
    }
    return d + __shfl_xor_sync(0xffffffffu, d, 1);
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

// Stage block [k0, k0 + BK) of a tile of `rows` rows from row0 on (what lies
// outside the operand or at or past kend reads as zero), the share of part
// `part` of `parts` warps: eight lanes per line, one 16-byte chunk each.  A
// line stays within 128 bytes of shared memory: with its chunks spread over
// the tile (the unswizzled layout) each 32-byte sector that arrives is split
// (17,920 x 64 x 384: 22.5 us against 16.5 at otherwise the same code).
template <bool MN>
__device__ __forceinline__ void stage_tile(uint32_t smem, const Operand& o, int row0, int rows, int k0,
                                           int kend, int part, int parts) {
    const int lane = threadIdx.x & 31, c = lane & 7;
    const int nlines = MN ? BK : rows;
    const int line0 = MN ? k0 : row0;
    const int left = (MN ? min(kend, o.lines) : o.lines) - line0;  // lines that exist
    const int i0 = part * 4 + (lane >> 3), step = 4 * parts;
    for (int blk = 0; blk < (MN ? rows : 1); blk += 64) {
        if (MN && blk + c * 8 >= rows) break;  // never read by the MMA
        const int col = (MN ? row0 + blk : k0) + c * 8;
        const bool cin = col < (MN ? o.cols : kend);
        const uint32_t dst = smem + (MN ? blk * (BK * 2) : 0);
        if (o.lout == 0) {
            const uint16_t* src = o.p + (size_t)(line0 + i0) * o.ld + col;
            const size_t inc = (size_t)step * o.ld;
#pragma unroll 4
            for (int i = i0; i < nlines; i += step, src += inc) {
                const bool ok = cin && i < left;
                cp16(dst + i * 128 + ((c ^ (i & 7)) << 4), ok ? src : o.p, ok);
            }
        } else {
            int n = (line0 + i0) / o.lout, l = (line0 + i0) - n * o.lout;
            for (int i = i0; i < nlines; i += step) {
                const int e = o.off + l * o.ld + col;
                const bool ok = cin && i < left && (unsigned)e < (unsigned)o.batch;
                cp16(dst + i * 128 + ((c ^ (i & 7)) << 4), ok ? o.p + (size_t)n * o.batch + e : o.p, ok);
                for (l += step; l >= o.lout; l -= o.lout) ++n;
            }
        }
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
template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(NT, 1) gemm_kernel(const GemmArgs g) {
    extern __shared__ uint8_t smem[];
    __shared__ uint64_t s_full[STAGES_MAX], s_free[STAGES_MAX];
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_ok;
    __shared__ int s_drained;
    __shared__ float s_col[4][BN_MAX];
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
    const int stage_bytes = tile_bytes(BM) + (B_MN ? mn_tile_bytes(bn) : tile_bytes(bn));
    const uint32_t full0 = smem_u32(&s_full[0]), free0 = smem_u32(&s_free[0]);
    const int log_s = 31 - __clz(S);

    // Stage kb % S holds block kb; its loads complete phase kb / S of the
    // stage's "full" barrier, its MMAs phase kb / S of its "free" barrier.
    if (warp < LOADERS) {
        const int st = warp / parts, part = warp - st * parts;
        const uint32_t sA = base + st * stage_bytes, sB = sA + tile_bytes(BM);
        const uint32_t full = full0 + 8 * st, freed = free0 + 8 * st;
        for (int kb = st; kb < nkb; kb += S) {
            // one decision for the warp: each lane probes and reads the clock by
            // itself, and at the limit they may disagree
            const bool freed_ok = kb < S || mbar_wait(freed, (uint32_t)(((kb >> log_s) - 1) & 1), g.wait_ns);
            if (!freed_ok) s_ok = 0;
            if (!__all_sync(0xffffffffu, freed_ok && s_ok)) break;
            const int k0 = kbeg + kb * BK;
            stage_tile<A_MN>(sA, g.A, m0, BM, k0, kend, part, parts);
            stage_tile<B_MN>(sB, g.B, n0, bn, k0, kend, part, parts);
            asm volatile("cp.async.wait_all;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(full);
        }
    } else {
        // The whole warp walks the K loop (uniform control flow and operands;
        // one thread in a divergent branch took 1,150 cycles a block, twice
        // the loads' share) and one elected lane issues.
        const uint32_t idesc = instr_desc(bn, A_MN, B_MN);
        const uint64_t descA = smem_desc(base, A_MN), descB = smem_desc(base + tile_bytes(BM), B_MN);
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
                        mma_bf16(tmem, ad + k_step<A_MN>() * t, bd + k_step<B_MN>() * t, idesc,
                                 (kb > 0 || t > 0) ? 1u : 0u);
                } else {
                    for (int t = 0; t * 16 < ktail; ++t)
                        mma_bf16(tmem, ad + k_step<A_MN>() * t, bd + k_step<B_MN>() * t, idesc,
                                 (kb > 0 || t > 0) ? 1u : 0u);
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
            if (g.adj_pre) {
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const bool in = r < g.M && n0 + c0 + i < g.N;
                    v[i] = in ? v[i] * gelu_grad(g.adj_pre[(size_t)r * g.ldc + n0 + c0 + i]) : 0.0f;
                }
                const float sum = column_sum16(v);
                if ((lane & 1) == 0) s_col[warp & 3][c0 + (lane >> 1)] = sum;
            }
            if (r < g.M) epilogue16(g, r, n0 + c0, v, vec);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (ok && g.adj_pre && tid < bn && n0 + tid < g.N)  // the four row quarters, in order
        g.colpart[(size_t)blockIdx.x * g.N + n0 + tid] =
            ((s_col[0][tid] + s_col[1][tid]) + s_col[2][tid]) + s_col[3][tid];
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

// p_bf16, if given, receives the updated parameters rounded to bf16.
__global__ void adam_kernel(float* p, const float* g, float* m, float* v, long long count, float lr,
                            float b1, float b2, float eps, float c1, float c2, uint16_t* p_bf16) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count;
         i += (long long)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        p[i] = pi;
        if (p_bf16) p_bf16[i] = f_to_bf16(pi);
    }
}

int grid_for(long long n, int threads) {
    long long b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    return (int)(b > 148LL * 16 ? 148LL * 16 : b);
}

// ------------------------------------------------------ network kernels
// im2col of the fp32 network input, eight columns (one 16-byte store) per
// thread (one element per thread, 64-bit index divisions: 22 us for the
// first layer of 256 records; this form 8 us).
__global__ void im2col8_kernel(const float* __restrict__ x, int Nb, int Lin, int Cin, int sn, int sl, int sc,
                               int k, int stride, int pad, int Lout, float scale, uint16_t* cols, int ldcols) {
    const unsigned per = (unsigned)ldcols / 8, total = (unsigned)Nb * Lout * per;
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const unsigned row = t / per;
    const int c0 = (int)(t - row * per) * 8;
    const int n = (int)(row / (unsigned)Lout), l0 = (int)(row - (unsigned)n * Lout) * stride - pad;
    int kk = c0 / Cin, ci = c0 - kk * Cin;
    uint16_t v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int l = l0 + kk;
        float f = 0.0f;
        if (kk < k && l >= 0 && l < Lin) f = x[(size_t)n * sn + (size_t)l * sl + (size_t)ci * sc] * scale;
        v[e] = f_to_bf16(f);
        if (++ci == Cin) {
            ci = 0;
            ++kk;
        }
    }
    uint4 q;
    q.x = v[0] | (uint32_t)v[1] << 16;
    q.y = v[2] | (uint32_t)v[3] << 16;
    q.z = v[4] | (uint32_t)v[5] << 16;
    q.w = v[6] | (uint32_t)v[7] << 16;
    *reinterpret_cast<uint4*>(cols + (size_t)row * ldcols + c0) = q;
}

constexpr int ADJ_ROWS = 128, ADJ_COLS = 1024;  // rows and channels per block of the kernel below
dim3 adjoint_rows_grid(int rows, int C) {
    return dim3((rows + ADJ_ROWS - 1) / ADJ_ROWS, (C + ADJ_COLS - 1) / ADJ_COLS);
}

// Adjoint of a layer's activation over [rows, C], four channels per thread:
// the adjoint of the activation is src itself (k == 0) or gathered from the
// next convolution's patches (the sum of nn_col2im, in its order); times
// gelu'(pre) if pre is given; written as bf16, with the column sums of each
// block's rows (the bias gradient's partial sums).  One pass in place of
// col2im, activation adjoint, transpose and column sums, with three fp32
// arrays written and read back (first convolution of 256 records: 120 us in
// four kernels, 12 us here; memory bound, 32 MB).  A block's 256 threads
// share the rows of up to 1,024 channels (blockIdx.y: which); where C / 4
// does not divide 256 the threads past the last whole row idle.
__global__ void __launch_bounds__(256) adjoint_rows_kernel(const float* __restrict__ src, int ld, int rows, int C,
                                                           int Lin, int k, int stride, int pad, int Lout,
                                                           const float* __restrict__ pre, uint16_t* d_bf16,
                                                           float* colpart) {
    __shared__ float4 s_sum[256];
    const int c0 = blockIdx.y * ADJ_COLS;
    const int tpr = min(C - c0, ADJ_COLS) / 4, rpp = 256 / tpr;  // threads per row, rows per pass
    const int t = threadIdx.x, g = t / tpr, c = c0 + (t - g * tpr) * 4;
    float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int row0 = blockIdx.x * ADJ_ROWS, row1 = g < rpp ? min(rows, row0 + ADJ_ROWS) : 0;
    for (int r = row0 + g; r < row1; r += rpp) {
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (k == 0) {  // (the caller's array: any alignment)
            const float* q = src + (size_t)r * ld + c;
            v = make_float4(q[0], q[1], q[2], q[3]);
        } else {
            const int n = r / Lin, l = r - n * Lin;
            for (int kk = (l + pad) % stride; kk < k; kk += stride) {  // kk = l + pad - lo * stride
                const int lo = (l + pad - kk) / stride;
                if (l + pad < kk || lo >= Lout) continue;
                const float4 q =
                    *reinterpret_cast<const float4*>(src + ((size_t)n * Lout + lo) * ld + (size_t)kk * C + c);
                v.x += q.x;
                v.y += q.y;
                v.z += q.z;
                v.w += q.w;
            }
        }
        const size_t o = (size_t)r * C + c;
        if (pre) {
            const float4 q = *reinterpret_cast<const float4*>(pre + o);
            v.x *= gelu_grad(q.x);
            v.y *= gelu_grad(q.y);
            v.z *= gelu_grad(q.z);
            v.w *= gelu_grad(q.w);
        }
        ushort4 b;
        b.x = f_to_bf16(v.x);
        b.y = f_to_bf16(v.y);
        b.z = f_to_bf16(v.z);
        b.w = f_to_bf16(v.w);
        *reinterpret_cast<ushort4*>(d_bf16 + o) = b;
        sum.x += v.x;
        sum.y += v.y;
        sum.z += v.z;
        sum.w += v.w;
    }
    s_sum[t] = sum;
    __syncthreads();
    if (t < tpr) {
        for (int q = 1; q < rpp; ++q) {
            const float4 v = s_sum[q * tpr + t];
            sum.x += v.x;
            sum.y += v.y;
            sum.z += v.z;
            sum.w += v.w;
        }
        *reinterpret_cast<float4*>(colpart + (size_t)blockIdx.x * C + c) = sum;
    }
}

// Bias gradients of all layers: out[c] = sum of part[t][c], t < T, a warp per
// column (lanes stride over t, then a fixed tree).
constexpr int MAX_LAYERS = 8;
struct BiasArgs {
    const float* part[MAX_LAYERS];
    float* out[MAX_LAYERS];
    int T[MAX_LAYERS], n[MAX_LAYERS];
    int layers;
};

__global__ void bias_reduce_kernel(const BiasArgs a) {
    int c = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)), i = 0;
    while (i < a.layers && c >= a.n[i]) c -= a.n[i++];
    if (i == a.layers) return;
    const float* p = a.part[i] + c;
    float v = 0.0f;
    for (int t = threadIdx.x & 31; t < a.T[i]; t += 32) v += p[(size_t)t * a.n[i]];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0) a.out[i][c] = v;
}

// Dynamic shared memory limit raised once per device and kernel.
template <bool A_MN, bool B_MN>
int allow_smem() {
    static std::atomic<uint64_t> set{0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return SWE_ECUDA;
    if (set.load(std::memory_order_acquire) >> dev & 1) return SWE_OK;
    if (cudaFuncSetAttribute(gemm_kernel<A_MN, B_MN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             SMEM_MAX + SMEM_ALIGN) != cudaSuccess)
        return SWE_ECUDA;
    set.fetch_or(1ull << dev, std::memory_order_release);
    return SWE_OK;
}

// Launch the product of g's operands (everything but the launch shape is
// set), K split over ksplit CTAs at most.
template <bool A_MN, bool B_MN>
int launch_gemm(GemmArgs g, int ksplit, float* workspace, cudaStream_t s) {
    const int rc = allow_smem<A_MN, B_MN>();
    if (rc != SWE_OK) return rc;
    // K per split, a multiple of BK
    const int kblocks = (g.K + BK - 1) / BK;
    const int per = (kblocks + ksplit - 1) / ksplit;
    g.kchunk = per * BK;
    const int zs = (kblocks + per - 1) / per;
    g.partial = zs > 1 ? workspace : nullptr;
    // Tile columns: the widest tile (A is read once per column tile) whose
    // grid still has a CTA for each SM, or the narrowest.
    int bn = BN_MAX;
    const long long mz = (long long)((g.M + BM - 1) / BM) * zs;
    while (bn > 16 && (bn / 2 >= g.N || mz * ((g.N + bn - 1) / bn) < 148)) bn /= 2;
    g.bn = bn;
    const int stage = tile_bytes(BM) + (B_MN ? mn_tile_bytes(bn) : tile_bytes(bn));
    g.stages = 1;  // a power of two, no more than the K blocks need
    while (g.stages < per && g.stages < (bn == BN_MAX ? 4 : STAGES_MAX)) g.stages *= 2;
    const dim3 grid((g.M + BM - 1) / BM, (g.N + bn - 1) / bn, zs);
    gemm_kernel<A_MN, B_MN><<<grid, NT, std::max(g.stages * stage + SMEM_ALIGN, SMEM_MIN), s>>>(g);
    if (zs > 1) splitk_epilogue_kernel<<<grid_for((long long)g.M * g.N, 256), 256, 0, s>>>(g, zs);
    return cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

Operand lines(const uint16_t* p, int ld, int n, int cols) { return Operand{p, ld, n, cols, 0, 0, 0}; }

// ------------------------------------------------------------- the network
int round_up(int x, int m) { return (x + m - 1) / m * m; }
size_t align256(size_t x) { return (x + 255) / 256 * 256; }
int rows_of(const nn_layer& l, int nb) { return l.conv ? nb * l.lout : nb; }
int split_of(int K) { return K / 2048 < 1 ? 1 : (K / 2048 > 128 ? 128 : K / 2048); }

// The layer list that the functions below accept: convolutions (the first
// one on the fp32 input, the others in place on the previous layer's NLC
// activations), then dense layers.
bool valid_layers(const nn_layer* L, int n, int nb) {
    if (!L || n < 2 || n > MAX_LAYERS || nb < 1 || !L[0].conv || L[n - 1].conv) return false;
    for (int i = 0; i < n; ++i) {
        const nn_layer& l = L[i];
        if (l.cin < 1 || l.cout < 1 || l.kpad < 16 || l.kpad % 16 || l.w < 0 || l.b < 0 || l.w % 8) return false;
        if (l.conv) {
            if (i > 0 && !L[i - 1].conv) return false;
            if (l.k < 1 || l.stride < 1 || l.pad < 0 || l.lin < 1 ||
                l.lout != (l.lin + 2 * l.pad - l.k) / l.stride + 1 || l.lout < 1 || l.kpad < l.k * l.cin)
                return false;
            if (i > 0 && (l.cin != L[i - 1].cout || l.lin != L[i - 1].lout || l.kpad != l.k * l.cin)) return false;
        } else if (l.kpad != l.cin || l.cin != (L[i - 1].conv ? L[i - 1].cout * L[i - 1].lout : L[i - 1].cout)) {
            return false;
        }
        // rows of 16-byte chunks; 32-bit row numbers and places within a record
        if (i + 1 < n && l.cout % 16) return false;
        const long long per = l.conv ? l.lout : 1;
        if (nb * per > (1ll << 30) || per * std::max(l.kpad, l.cout) >= (1ll << 31)) return false;
    }
    return true;
}

// Workspace of one batch size: forward buffers, then the backward ones.
struct NetBuffers {
    uint16_t* cols;                 // first layer's patches
    float* pre[MAX_LAYERS];         // pre-activations
    uint16_t* act[MAX_LAYERS];      // activations (not of the last layer)
    uint16_t* d[MAX_LAYERS];        // adjoints of the pre-activations
    float* dcols;                   // adjoint of a convolution's patches
    float* colpart[MAX_LAYERS];     // column sums of d, per row tile
    float* split;                   // partial products
    size_t bytes;
};

int column_tiles(const nn_layer* L, int n, int i, int nb) {
    // the last layer and the inputs of convolutions: adjoint_rows_kernel; the
    // others: the row tiles of the product that makes them
    const int rows = rows_of(L[i], nb);
    if (i == n - 1 || L[i + 1].conv) return (rows + ADJ_ROWS - 1) / ADJ_ROWS;
    return (nb + BM - 1) / BM * (rows / nb);
}

NetBuffers carve(void* ws, const nn_layer* L, int n, int nb, bool training) {
    NetBuffers b{};
    size_t at = 0;
    auto take = [&](size_t bytes) {
        void* p = static_cast<char*>(ws) + at;
        at += align256(bytes);
        return p;
    };
    b.cols = (uint16_t*)take((size_t)nb * L[0].lout * L[0].kpad * 2);
    for (int i = 0; i < n; ++i) {
        const size_t e = (size_t)rows_of(L[i], nb) * L[i].cout;
        b.pre[i] = (float*)take(e * 4);
        if (i + 1 < n) b.act[i] = (uint16_t*)take(e * 2);
    }
    if (training) {
        size_t dc = 0, sp = 0;
        for (int i = 0; i < n; ++i) {
            const int rows = rows_of(L[i], nb), Mp = round_up(rows, 64);
            b.d[i] = (uint16_t*)take((size_t)rows * L[i].cout * 2);
            b.colpart[i] = (float*)take((size_t)column_tiles(L, n, i, nb) * L[i].cout * 4);
            if (i > 0 && L[i].conv) dc = std::max(dc, (size_t)rows * L[i].kpad * 4);
            if (split_of(Mp) > 1) sp = std::max(sp, (size_t)split_of(Mp) * L[i].cout * L[i].kpad * 4);
        }
        b.dcols = (float*)take(dc);
        b.split = (float*)take(sp);
    }
    b.bytes = at;
    return b;
}

// Layer i's input as lines of its data rows.
Operand layer_input(const nn_layer* L, const NetBuffers& b, int i, int nb) {
    const nn_layer& l = L[i];
    if (i == 0) return lines(b.cols, l.kpad, nb * l.lout, l.kpad);
    if (!l.conv) return lines(b.act[i - 1], l.cin, nb, l.cin);
    return Operand{b.act[i - 1], l.stride * l.cin, nb * l.lout, l.kpad, l.lout, l.lin * l.cin, -l.pad * l.cin};
}

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
    GemmArgs g{};
    g.A = lines(A, lda, M, K);
    g.B = lines(B, ldb, N, K);
    g.M = M;
    g.N = N;
    g.K = K;
    g.bias = bias;
    g.act = act;
    g.ldc = ldc;
    g.out_f32 = out_f32;
    g.out_bf16 = out_bf16;
    g.pre_f32 = pre_f32;
    g.err = err;
    g.wait_ns = (unsigned long long)wait_ns;
    return launch_gemm<false, false>(g, ksplit, workspace, (cudaStream_t)stream);
}

extern "C" long long nn_net_workspace_bytes(const nn_layer* layers, int nlayers, int nb, int training) {
    if (!valid_layers(layers, nlayers, nb)) return -1;
    return (long long)carve(nullptr, layers, nlayers, nb, training != 0).bytes;
}

extern "C" int nn_net_forward(const nn_layer* layers, int nlayers, const float* params,
                              const uint16_t* params_bf16, const float* x, float in_scale, int nb,
                              void* workspace, float* out, long long wait_ns, uint32_t* err, void* stream) {
    if (!valid_layers(layers, nlayers, nb) || !params || !params_bf16 || !x || !workspace || !out || wait_ns < 0)
        return SWE_EARG;
    if (((uintptr_t)workspace & 255u) || ((uintptr_t)params_bf16 & 15u)) return SWE_EARG;
    cudaStream_t s = (cudaStream_t)stream;
    const nn_layer* L = layers;
    const NetBuffers b = carve(workspace, L, nlayers, nb, false);
    {
        const nn_layer& l = L[0];  // x is [nb, cin, lin]
        const long long per = (long long)l.lout * (l.kpad / 8);  // the kernel's indices are 32-bit
        const int step = (int)std::max(1ll, std::min((long long)nb, (1ll << 31) / per));
        for (int n0 = 0; n0 < nb; n0 += step) {
            const int count = std::min(step, nb - n0);
            im2col8_kernel<<<(unsigned)((count * per + 255) / 256), 256, 0, s>>>(
                x + (size_t)n0 * l.cin * l.lin, count, l.lin, l.cin, l.cin * l.lin, 1, l.lin, l.k, l.stride, l.pad,
                l.lout, in_scale, b.cols + (size_t)n0 * l.lout * l.kpad, l.kpad);
        }
    }
    for (int i = 0; i < nlayers; ++i) {
        const nn_layer& l = L[i];
        const bool last = i == nlayers - 1;
        GemmArgs g{};
        g.A = layer_input(L, b, i, nb);
        g.B = lines(params_bf16 + l.w, l.kpad, l.cout, l.kpad);
        g.M = rows_of(l, nb);
        g.N = l.cout;
        g.K = l.kpad;
        g.bias = params + l.b;
        g.act = last ? NN_ACT_NONE : NN_ACT_GELU;
        g.ldc = l.cout;
        g.out_f32 = last ? out : nullptr;
        g.out_bf16 = last ? nullptr : b.act[i];
        g.pre_f32 = b.pre[i];
        g.err = err;
        g.wait_ns = (unsigned long long)wait_ns;
        const int rc = launch_gemm<false, false>(g, 1, nullptr, s);
        if (rc != SWE_OK) return rc;
    }
    return cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

extern "C" int nn_net_backward(const nn_layer* layers, int nlayers, const uint16_t* params_bf16,
                               const float* dout, int nb, void* workspace, float* grads,
                               long long wait_ns, uint32_t* err, void* stream) {
    if (!valid_layers(layers, nlayers, nb) || !params_bf16 || !dout || !workspace || !grads || wait_ns < 0)
        return SWE_EARG;
    const nn_layer* L = layers;
    const int n = nlayers;
    if (L[n - 1].cout % 16) return SWE_EARG;
    if (((uintptr_t)workspace & 255u) || ((uintptr_t)params_bf16 & 15u)) return SWE_EARG;
    cudaStream_t s = (cudaStream_t)stream;
    const NetBuffers b = carve(workspace, L, n, nb, true);
    BiasArgs ba{};
    int columns = 0;
    ba.layers = n;
    for (int i = 0; i < n; ++i) {
        ba.part[i] = b.colpart[i];
        ba.out[i] = grads + L[i].b;
        ba.T[i] = column_tiles(L, n, i, nb);
        ba.n[i] = L[i].cout;
        columns += L[i].cout;
    }
    adjoint_rows_kernel<<<adjoint_rows_grid(nb, L[n - 1].cout), 256, 0, s>>>(
        dout, L[n - 1].cout, nb, L[n - 1].cout, 0, 0, 0, 0, 0, nullptr, b.d[n - 1], b.colpart[n - 1]);
    for (int i = n - 1; i >= 0; --i) {
        const nn_layer& l = L[i];
        const int rows = rows_of(l, nb), Mp = round_up(rows, 64);
        GemmArgs g{};
        g.err = err;
        g.wait_ns = (unsigned long long)wait_ns;
        // dW [cout, kpad] = d^T X: both operands read in place, a line per data row
        g.A = lines(b.d[i], l.cout, rows, l.cout);
        g.B = layer_input(L, b, i, nb);
        g.M = l.cout;
        g.N = g.ldc = l.kpad;
        g.K = Mp;
        g.out_f32 = grads + l.w;
        int rc = launch_gemm<true, true>(g, split_of(Mp), b.split, s);
        if (rc != SWE_OK) return rc;
        if (i == 0) break;
        // dX [rows, kpad] = d W
        g.A = lines(b.d[i], l.cout, rows, l.cout);
        g.B = lines(params_bf16 + l.w, l.kpad, l.cout, l.kpad);
        g.M = rows;
        g.N = g.ldc = l.kpad;
        g.K = l.cout;
        g.out_f32 = nullptr;
        if (!l.conv) {  // straight to the adjoint of the previous pre-activations
            g.adj_pre = b.pre[i - 1];
            g.out_bf16 = b.d[i - 1];
            g.colpart = b.colpart[i - 1];
            rc = launch_gemm<false, true>(g, 1, nullptr, s);
            if (rc != SWE_OK) return rc;
        } else {
            g.out_f32 = b.dcols;
            rc = launch_gemm<false, true>(g, 1, nullptr, s);
            if (rc != SWE_OK) return rc;
            const int prows = nb * l.lin;
            adjoint_rows_kernel<<<adjoint_rows_grid(prows, l.cin), 256, 0, s>>>(
                b.dcols, l.kpad, prows, l.cin, l.lin, l.k, l.stride, l.pad, l.lout, b.pre[i - 1], b.d[i - 1],
                b.colpart[i - 1]);
        }
    }
    bias_reduce_kernel<<<(columns + 7) / 8, 256, 0, s>>>(ba);
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

extern "C" int nn_adam_bf16(float* params, const float* grads, float* m, float* v, long long count, float lr,
                            float beta1, float beta2, float eps, int step, uint16_t* params_bf16, void* stream) {
    if (!params || !grads || !m || !v || count < 1 || step < 1) return SWE_EARG;
    const float c1 = 1.0f - powf(beta1, (float)step);
    const float c2 = 1.0f - powf(beta2, (float)step);
    adam_kernel<<<grid_for(count, 256), 256, 0, (cudaStream_t)stream>>>(params, grads, m, v, count, lr, beta1,
                                                                        beta2, eps, c1, c2, params_bf16);
    return cudaGetLastError() == cudaSuccess ? SWE_OK : SWE_ECUDA;
}

extern "C" int nn_adam(float* params, const float* grads, float* m, float* v, long long count, float lr,
                       float beta1, float beta2, float eps, int step, void* stream) {
    return nn_adam_bf16(params, grads, m, v, count, lr, beta1, beta2, eps, step, nullptr, stream);
}

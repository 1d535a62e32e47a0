// INT4-AWQ GEMM on the 5th-generation tensor cores (tcgen05 + TMEM) for calls of many token rows:
// prefill chunks and batched decode, where the operation is a dense contraction.
// Same placeholder as the GEMV: kuiper/include/op/matmul.h:1-11 of the reference.
//
// y[M,N] (+)= x[M,K] . dequant(qweight)[K,N]
//
// Calls of up to 32 rows go to awq_gemm_rows.cu, others to the 256 x 256 tiles of awq_gemm_tc4_kernel further down; the two
// kernels described first remain for what those do not take (N % 32 != 0, no K split wanted, see tiles_pay).
//
// One CTA owns a 128 x 256 output tile; its fp32 accumulator lives in tensor memory (128 lanes x 256
// columns), two CTAs share an SM.  The activations are converted to fp16 once per call (the same operand
// rounding as the GEMV) and reach shared memory with cp.async; every thread dequantises one packed word
// column and one K octet of the weight tile: the nibble pairs come out of the LOP3 / 0x6400 trick exactly
// as in the GEMV, the fp16 group scale is applied, and register transposes (PRMT) turn "two columns of one
// row" into "two rows of one column", so that each column's eight K values are one 16-byte shared-memory
// store.  Both operands are stored K-major with the 128-byte swizzle: a tile row is the 64 K values (128
// bytes) of one token row / weight column, eight rows form a 1024-byte atom, and the 16-byte chunk c of row
// r sits at chunk position c ^ (r % 8).  One thread issues four tcgen05.mma (K = 16 each) per stage and a
// tcgen05.commit onto the stage's mbarrier; a stage is refilled only after that commit.  In
// awq_gemm_tc3_kernel that thread belongs to a warp of its own and learns through a second mbarrier that the
// producer warps have filled the stage; awq_gemm_tc2_kernel hands the stage over at a block-wide barrier.  The
// epilogue reads the accumulator with tcgen05.ld (one TMEM lane = one output row per thread).
//
// Every mbarrier wait is bounded; on a timeout the CTA records an error word, stops issuing work,
// still frees its tensor memory and returns.
#include <cuda.h>
#include <cstring>

#include "common.cuh"

namespace kuiper {
namespace {

constexpr int kBM = 128, kBK = 64;
constexpr int kGemmThreads = 256;
constexpr uint32_t kMagicTc = 0x64006400u;
constexpr int kSpinLimitTc = 1 << 22;  // polls of one wait, about a microsecond each

__device__ int g_gemm_wait_error = 0;

constexpr uint32_t kDescLayoutSw128 = 2;  // layout field of the matrix descriptor: 128-byte swizzle
constexpr uint32_t kDescVersion = 1;

struct GemmParams {
    const float* x;        // [M, K]
    const uint32_t* qw;    // [K, N/8]
    const uint32_t* qz;    // [K/128, N/8]
    const __half* scales;  // [K/128, N]
    float* y;              // [M, N]
    const float* residual; // mode 1
    int M, K, N;
    int mode;              // 0: y = acc, 1: y = acc + residual, 2: y += acc
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ __half2 tc_u2h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
__device__ __forceinline__ uint32_t tc_h22u(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }

__device__ __forceinline__ bool tc_mbar_wait(uint64_t* bar, uint32_t parity, int spins = kSpinLimitTc) {
    const uint32_t addr = smem_addr(bar);
    for (int spin = 0; spin < spins; spin++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// 64-bit shared-memory matrix descriptor: start address, leading / stride byte offsets (all >> 4),
// descriptor version, swizzle mode
// K-major, 128-byte swizzle: 8-row atoms are 1024 B apart; the leading offset is unused because one
// atom spans the whole K tile
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= uint64_t((saddr >> 4) & 0x3fffu);
    d |= uint64_t((1024u >> 4) & 0x3fffu) << 32;
    d |= uint64_t(kDescVersion) << 46;
    d |= uint64_t(kDescLayoutSw128) << 61;
    return d;
}

struct TileConsts {
    __half2 z0, z1, z2, z3;  // (1024 + z) pairs for the low nibbles, -(64 + z) pairs for the high nibbles
    __half2 s0, s1, s2, s3;  // fp16 scales of column pairs (0,1) (2,3) (4,5) (6,7)
};
__device__ __forceinline__ TileConsts make_tile_consts(uint32_t zw, const uint4& sraw) {
    const __half2 neg_sixteenth = __floats2half2_rn(-0.0625f, -0.0625f);
    const uint32_t z8 = zw >> 8;
    TileConsts c;
    c.z0 = tc_u2h2((zw & 0x000f000fu) | kMagicTc);
    c.z1 = __hmul2(tc_u2h2((zw & 0x00f000f0u) | kMagicTc), neg_sixteenth);
    c.z2 = tc_u2h2((z8 & 0x000f000fu) | kMagicTc);
    c.z3 = __hmul2(tc_u2h2((z8 & 0x00f000f0u) | kMagicTc), neg_sixteenth);
    c.s0 = tc_u2h2(sraw.x); c.s1 = tc_u2h2(sraw.y); c.s2 = tc_u2h2(sraw.z); c.s3 = tc_u2h2(sraw.w);
    return c;
}
__device__ __forceinline__ void dequant_word_consts(uint32_t w, const TileConsts& c, uint32_t (&out)[4]) {
    const __half2 sixteenth = __floats2half2_rn(0.0625f, 0.0625f);
    const uint32_t w8 = w >> 8;
    out[0] = tc_h22u(__hmul2(__hsub2(tc_u2h2((w & 0x000f000fu) | kMagicTc), c.z0), c.s0));
    out[1] = tc_h22u(__hmul2(__hfma2(tc_u2h2((w & 0x00f000f0u) | kMagicTc), sixteenth, c.z1), c.s1));
    out[2] = tc_h22u(__hmul2(__hsub2(tc_u2h2((w8 & 0x000f000fu) | kMagicTc), c.z2), c.s2));
    out[3] = tc_h22u(__hmul2(__hfma2(tc_u2h2((w8 & 0x00f000f0u) | kMagicTc), sixteenth, c.z3), c.s3));
}

// ---------------------------------------------------------------------------------------------
// Second generation: 128 x 256 tiles, two CTAs per SM, no global-memory latency on the critical path.
//   * the activations are converted to fp16 once per call (convert_f16_kernel) and reach shared memory with
//     cp.async, 16 bytes per (row, K octet), straight into their swizzled position, one tile ahead;
//   * the packed weights of the next tile are already in registers while the current tile is dequantised;
//   * a stage is reused only after the tcgen05.commit of the MMAs that read it; two stages of 48 KB, so that two
//     CTAs share an SM and one's dequantisation overlaps the other's MMAs.
constexpr int kBN2 = 256;
constexpr int kStages2 = 2;   // 96 KB per CTA: two CTAs (16 warps, 2 x 256 TMEM columns) share an SM
constexpr int kStageA2 = kBM * kBK * 2;   // 16 KB
constexpr int kStageB2 = kBN2 * kBK * 2;  // 32 KB

// x -> fp16 copy; optionally zeroes the output of a split-K call (zero4 float4s), so that the zeroing is a kernel of
// the programmatic-dependent-launch chain like everything else (the GEMM's dependency wait covers it)
__global__ void convert_f16_kernel(const float4* __restrict__ x, uint2* __restrict__ out, int64_t n4, float4* __restrict__ zero,
                                   int64_t zero4) {
    pdl_launch_dependents();
    pdl_wait();
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n4; i += stride) {
        const float4 v = __ldcg(x + i);
        out[i] = make_uint2(tc_h22u(__floats2half2_rn(v.x, v.y)), tc_h22u(__floats2half2_rn(v.z, v.w)));
    }
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < zero4; i += stride) zero[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

struct GemmParams2 {
    GemmParams g;
    const __half* x16;  // [M, K] fp16 copy of x
    int tiles_per_split; // third generation: 64-row K tiles of one CTA (grid.z CTAs share an output tile); 0 = all of K
};

__global__ void __launch_bounds__(kGemmThreads, 2) awq_gemm_tc2_kernel(const GemmParams2 pp) {
    const GemmParams& p = pp.g;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);
    unsigned char* sA = smem;                          // kStages2 x 16 KB
    unsigned char* sB = smem + kStages2 * kStageA2;    // kStages2 x 32 KB
    __shared__ uint64_t mma_bar[kStages2];
    __shared__ uint32_t s_tmem;
    __shared__ int s_dead;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.x * kBN2, m0 = blockIdx.y * kBM;
    const int NW = p.N >> 3;

    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < kStages2; i++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&mma_bar[i])));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_dead = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)), "r"(uint32_t(kBN2))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;

    pdl_launch_dependents();
    pdl_wait();

    const uint32_t idesc = (1u << 4) | (uint32_t(kBN2 >> 3) << 17) | (uint32_t(kBM >> 4) << 24);
    const int nk = p.K / kBK;
    bool dead = false;

    // ---- this thread's share of a tile; everything that does not depend on the tile is computed here
    // activations: four 16-byte chunks (row m, K octet koct), global fp16 -> swizzled shared memory
    const __half* a_src[4];
    uint32_t a_dst[4], a_bytes[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int item = q * kGemmThreads + tid;
        const int koct = item & 7, m = item >> 3;
        const bool ok = m0 + m < p.M;
        a_src[q] = pp.x16 + size_t(ok ? m0 + m : 0) * p.K + koct * 8;
        a_dst[q] = smem_addr(sA) + (m >> 3) * 1024 + (m & 7) * 128 + ((koct ^ (m & 7)) << 4);
        a_bytes[q] = ok ? 16u : 0u;  // 0: the chunk is zero filled
    }
    auto issue_a = [&](int tile, int stage) {
#pragma unroll
        for (int q = 0; q < 4; q++)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a_dst[q] + stage * kStageA2),
                         "l"(a_src[q] + tile * kBK), "r"(a_bytes[q])
                         : "memory");
    };
    // weights: packed word column j of the tile (8 output columns), K octet koct (8 rows)
    const int koct_b = tid & 7, j_b = tid >> 3;
    const int wcol = (n0 >> 3) + j_b;
    const bool col_ok = wcol < NW;
    const uint32_t* w_src = p.qw + (col_ok ? size_t(koct_b * 8) * NW + wcol : 0);  // + tile * kBK * NW + r * NW
    const uint32_t* z_src = p.qz + (col_ok ? wcol : 0);                            // + group * NW
    const uint4* s_src = reinterpret_cast<const uint4*>(p.scales + (col_ok ? n0 + j_b * 8 : 0));  // + group * N halves
    const int tile_words = kBK * NW;
    auto load_b = [&](int tile, uint32_t (&w)[8], uint32_t& zw, uint4& sraw) {
        const uint32_t* wp = w_src + size_t(tile) * tile_words;
        const int g = tile >> 1;  // two 64-row tiles per 128-row group
#pragma unroll
        for (int r = 0; r < 8; r++) w[r] = col_ok ? __ldg(wp + r * NW) : 0u;
        zw = col_ok ? __ldg(z_src + size_t(g) * NW) : 0u;
        sraw = col_ok ? __ldg(s_src + size_t(g) * (p.N >> 3)) : make_uint4(0, 0, 0, 0);
    };

    // one tile of the K loop; the packed words of tile `it` are in (w, zw, sraw) and the same registers are
    // refilled with tile it + 2 as soon as they have been consumed, so a load has two tiles of time to land
    auto tile_step = [&](int it, uint32_t (&w)[8], uint32_t& zw, uint4& sraw) {
        const int s = it % kStages2;
        // ---- dequantise the weight tile into stage s (free: checked one tile ago, when its activations were requested)
        {
            uint32_t d[8][4];  // [row][column pair]
            const TileConsts tc = make_tile_consts(zw, sraw);
#pragma unroll
            for (int r = 0; r < 8; r++) dequant_word_consts(w[r], tc, d[r]);
            if (it + 2 < nk) load_b(it + 2, w, zw, sraw);
            unsigned char* dst = sB + s * kStageB2 + j_b * 1024;
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const int pr = c >> 1;
                const uint32_t sel = (c & 1) ? 0x7632u : 0x5410u;
                uint4 o;  // rows (0,1) (2,3) (4,5) (6,7) of column c
                o.x = __byte_perm(d[0][pr], d[1][pr], sel);
                o.y = __byte_perm(d[2][pr], d[3][pr], sel);
                o.z = __byte_perm(d[4][pr], d[5][pr], sel);
                o.w = __byte_perm(d[6][pr], d[7][pr], sel);
                *reinterpret_cast<uint4*>(dst + c * 128 + ((koct_b ^ c) << 4)) = o;
            }
        }
        // ---- request the next tile's activations; its stage is free once the MMAs that last read it have finished
        //      (by now they had the whole dequantisation above to do so)
        if (it + 1 < nk) {
            const int sn = (it + 1) % kStages2;
            if (it + 1 >= kStages2 && !dead) {
                if (!tc_mbar_wait(&mma_bar[sn], uint32_t((it + 1) / kStages2 - 1) & 1u)) {
                    atomicExch(&g_gemm_wait_error, 3);
                    s_dead = 1;
                    dead = true;
                }
            }
            issue_a(it + 1, sn);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");  // everything but the newest group: this tile's activations
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        dead = dead || (s_dead != 0);
        if (tid == 0 && !dead) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a_base = smem_addr(sA + s * kStageA2), b_base = smem_addr(sB + s * kStageB2);
#pragma unroll
            for (int kk = 0; kk < kBK / 16; kk++) {
                const uint64_t adesc = make_desc(a_base + kk * 32);
                const uint64_t bdesc = make_desc(b_base + kk * 32);
                const uint32_t accumulate = (it > 0 || kk > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                    ::"r"(tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(&mma_bar[s]))
                         : "memory");
        }
    };

    uint32_t w_even[8], w_odd[8], zw_even, zw_odd = 0;
    uint4 s_even, s_odd = make_uint4(0, 0, 0, 0);
    issue_a(0, 0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    load_b(0, w_even, zw_even, s_even);
    if (nk > 1) load_b(1, w_odd, zw_odd, s_odd);
    for (int it = 0; it < nk; it += 2) {
        tile_step(it, w_even, zw_even, s_even);
        if (it + 1 < nk) tile_step(it + 1, w_odd, zw_odd, s_odd);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");

    // ---- all MMAs done?  (they complete in order: the last commit covers everything)
    if (!dead) {
        const int last = nk - 1;
        if (!tc_mbar_wait(&mma_bar[last % kStages2], uint32_t(last / kStages2) & 1u)) {
            atomicExch(&g_gemm_wait_error, 4);
            dead = true;
        }
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    if (!dead) {
        // ---- epilogue: warp w reads TMEM lanes 32*(w&3).., columns 128*(w>>2)..; one output row per thread
        const int row = m0 + (warp & 3) * 32 + lane;
        const int cbase = (warp >> 2) * 128;
#pragma unroll 1
        for (int ch = 0; ch < 4; ch++) {
            uint32_t r[32];
            const uint32_t taddr = tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t(cbase + ch * 32);
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                  "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
                  "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
                  "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                : "r"(taddr)
                : "memory");
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (row < p.M) {
                const int col0 = n0 + cbase + ch * 32;
                float* yp = p.y + size_t(row) * p.N + col0;
                const float* rp = p.mode == 1 ? p.residual + size_t(row) * p.N + col0 : (p.mode == 2 ? yp : nullptr);
#pragma unroll
                for (int v = 0; v < 8; v++) {
                    if (col0 + v * 4 < p.N) {
                        float4 o = make_float4(__uint_as_float(r[4 * v]), __uint_as_float(r[4 * v + 1]),
                                               __uint_as_float(r[4 * v + 2]), __uint_as_float(r[4 * v + 3]));
                        if (rp) {
                            const float4 a = __ldcg(reinterpret_cast<const float4*>(rp) + v);
                            o.x += a.x; o.y += a.y; o.z += a.z; o.w += a.w;
                        }
                        reinterpret_cast<float4*>(yp)[v] = o;
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(uint32_t(kBN2)) : "memory");
    }
}


// ---------------------------------------------------------------------------------------------
// Third generation: the same tiles, stages and dequantisation, but nobody waits at a block-wide barrier per stage.
//   * eight producer warps fill the stages (weights dequantised into stage s, activations of the next tile by cp.async);
//     each thread arrives on the stage's "full" mbarrier once its own copies have landed and its stores are visible to
//     the tensor-core proxy;
//   * a ninth warp only waits for "full", issues the four tcgen05.mma of the stage and commits them onto the stage's
//     "free" mbarrier, which the producers check before they overwrite the stage - so a producer warp that is ahead
//     keeps working on the next tile instead of waiting for the slowest warp of the block;
//   * zero words and scales are loaded and prepared once per 128-row group (two stages), addresses are carried as running
//     pointers, and the swizzled store offsets are computed once.
constexpr int kProducerThreads3 = 256;
constexpr int kGemmThreads3 = kProducerThreads3 + 32;

__global__ void __launch_bounds__(kGemmThreads3, 2) awq_gemm_tc3_kernel(const GemmParams2 pp) {
    const GemmParams& p = pp.g;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);
    unsigned char* sA = smem;                          // kStages2 x 16 KB
    unsigned char* sB = smem + kStages2 * kStageA2;    // kStages2 x 32 KB
    __shared__ uint64_t full_bar[kStages2];            // producers -> MMA warp
    __shared__ uint64_t free_bar[kStages2];            // tcgen05.commit -> producers
    __shared__ uint32_t s_tmem;
    __shared__ int s_dead;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.x * kBN2, m0 = blockIdx.y * kBM;
    const int NW = p.N >> 3;

    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < kStages2; i++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&full_bar[i])), "r"(uint32_t(kProducerThreads3)));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&free_bar[i])));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_dead = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)), "r"(uint32_t(kBN2))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;

    pdl_launch_dependents();
    pdl_wait();

    // split K: grid.z CTAs work on consecutive runs of K tiles of the same output tile and add their sums with reductions
    const int nk = pp.tiles_per_split > 0 ? pp.tiles_per_split : p.K / kBK;
    const int tile0 = int(blockIdx.z) * nk;
    const bool split_k = gridDim.z > 1;
    bool dead = false;

    if (warp == kProducerThreads3 / 32) {
        // ------------------------------------------------------------ MMA warp: one lane issues
        if (lane == 0) {
            const uint32_t idesc = (1u << 4) | (uint32_t(kBN2 >> 3) << 17) | (uint32_t(kBM >> 4) << 24);
            for (int it = 0; it < nk && !dead; it++) {
                const int s = it % kStages2;
                if (!tc_mbar_wait(&full_bar[s], uint32_t(it / kStages2) & 1u)) {
                    atomicExch(&g_gemm_wait_error, 5);
                    s_dead = 1;
                    dead = true;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a_base = smem_addr(sA + s * kStageA2), b_base = smem_addr(sB + s * kStageB2);
#pragma unroll
                for (int kk = 0; kk < kBK / 16; kk++) {
                    const uint64_t adesc = make_desc(a_base + kk * 32);
                    const uint64_t bdesc = make_desc(b_base + kk * 32);
                    const uint32_t accumulate = (it > 0 || kk > 0) ? 1u : 0u;
                    asm volatile(
                        "{\n\t.reg .pred p;\n\t"
                        "setp.ne.b32 p, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                        ::"r"(tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
                        : "memory");
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(&free_bar[s]))
                             : "memory");
            }
        }
    } else {
        // ------------------------------------------------------------ producers
        // activations: four 16-byte chunks (row m, K octet koct), global fp16 -> swizzled shared memory, one tile ahead
        const unsigned char* a_src[4];
        uint32_t a_dst[4], a_bytes[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int item = q * kProducerThreads3 + tid;
            const int koct = item & 7, m = item >> 3;
            const bool ok = m0 + m < p.M;
            a_src[q] = reinterpret_cast<const unsigned char*>(pp.x16 + size_t(ok ? m0 + m : 0) * p.K + koct * 8 + size_t(tile0) * kBK);
            a_dst[q] = smem_addr(sA) + (m >> 3) * 1024 + (m & 7) * 128 + ((koct ^ (m & 7)) << 4);
            a_bytes[q] = ok ? 16u : 0u;  // 0: the chunk is zero filled
        }
        auto issue_a = [&](int stage) {  // the next tile along K; the sources advance by one tile
#pragma unroll
            for (int q = 0; q < 4; q++) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a_dst[q] + stage * kStageA2), "l"(a_src[q]),
                             "r"(a_bytes[q])
                             : "memory");
                a_src[q] += kBK * sizeof(__half);
            }
        };
        // weights: packed word column j of the tile (8 output columns), K octet koct (8 rows)
        const int koct_b = tid & 7, j_b = tid >> 3;
        const int wcol = (n0 >> 3) + j_b;
        const bool col_ok = wcol < NW;
        const size_t tile_words = size_t(kBK) * NW;
        const size_t row_words = size_t(NW);
        const size_t scale_vecs = size_t(p.N >> 3);
        const size_t group0 = size_t(tile0 >> 1);  // a split starts at a 128-row group
        const uint32_t* w_next = p.qw + (col_ok ? size_t(koct_b * 8) * NW + wcol + size_t(tile0) * tile_words : 0);  // next tile to load
        const uint32_t* z_next = p.qz + (col_ok ? wcol + group0 * row_words : 0);       // zero word of the next group to load
        const uint4* s_next = reinterpret_cast<const uint4*>(p.scales + (col_ok ? n0 + j_b * 8 : 0)) + (col_ok ? group0 * scale_vecs : 0);
        auto load_w = [&](uint32_t (&w)[8]) {
#pragma unroll
            for (int r = 0; r < 8; r++) w[r] = col_ok ? __ldg(w_next + r * row_words) : 0u;
            w_next += tile_words;
        };
        auto load_consts = [&](uint32_t& zw, uint4& sraw) {
            zw = col_ok ? __ldg(z_next) : 0u;
            sraw = col_ok ? __ldg(s_next) : make_uint4(0, 0, 0, 0);
            z_next += row_words;
            s_next += scale_vecs;
        };
        // swizzled 16-byte store slots of this thread inside its 1024-byte column block
        uint32_t b_off[8];
#pragma unroll
        for (int c = 0; c < 8; c++) b_off[c] = uint32_t(c * 128 + ((koct_b ^ c) << 4));
        const uint32_t b_dst = smem_addr(sB) + j_b * 1024;

        TileConsts tc;
        auto tile_step = [&](int it, uint32_t (&w)[8]) {
            const int s = it % kStages2;
            {
                uint32_t d[8][4];  // [row][column pair]
#pragma unroll
                for (int r = 0; r < 8; r++) dequant_word_consts(w[r], tc, d[r]);
                if (it + 2 < nk) load_w(w);
                const uint32_t dst = b_dst + s * kStageB2;
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const int pr = c >> 1;
                    const uint32_t sel = (c & 1) ? 0x7632u : 0x5410u;
                    const uint32_t o0 = __byte_perm(d[0][pr], d[1][pr], sel), o1 = __byte_perm(d[2][pr], d[3][pr], sel);
                    const uint32_t o2 = __byte_perm(d[4][pr], d[5][pr], sel), o3 = __byte_perm(d[6][pr], d[7][pr], sel);
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + b_off[c]), "r"(o0), "r"(o1), "r"(o2), "r"(o3)
                                 : "memory");
                }
            }
            // the next tile's activations go into the other stage once the MMAs that last read it have finished
            if (it + 1 < nk) {
                const int sn = (it + 1) % kStages2;
                if (it + 1 >= kStages2 && !dead) {
                    if (!tc_mbar_wait(&free_bar[sn], uint32_t((it + 1) / kStages2 - 1) & 1u)) {
                        atomicExch(&g_gemm_wait_error, 3);
                        s_dead = 1;
                        dead = true;
                    }
                }
                issue_a(sn);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 1;" ::: "memory");  // everything but the newest group: this tile's activations
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&full_bar[s])) : "memory");
        };

        uint32_t w_even[8], w_odd[8], zw;
        uint4 sraw;
        issue_a(0);
        asm volatile("cp.async.commit_group;" ::: "memory");
        load_w(w_even);
        if (nk > 1) load_w(w_odd);
        load_consts(zw, sraw);
        for (int it = 0; it < nk; it += 2) {  // two 64-row tiles = one 128-row group: one set of constants
            tc = make_tile_consts(zw, sraw);
            if (it + 2 < nk) load_consts(zw, sraw);
            tile_step(it, w_even);
            if (it + 1 < nk) tile_step(it + 1, w_odd);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");

        // ---- all MMAs done?  (they complete in order: the last commit covers everything)
        if (!dead) {
            const int last = nk - 1;
            if (!tc_mbar_wait(&free_bar[last % kStages2], uint32_t(last / kStages2) & 1u)) {
                atomicExch(&g_gemm_wait_error, 4);
                dead = true;
            }
        }
        dead = dead || (s_dead != 0);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

        if (!dead) {
            // ---- epilogue: warp w reads TMEM lanes 32*(w&3).., columns 128*(w>>2)..; one output row per thread
            const int row = m0 + (warp & 3) * 32 + lane;
            const int cbase = (warp >> 2) * 128;
#pragma unroll 1
            for (int ch = 0; ch < 4; ch++) {
                uint32_t r[32];
                const uint32_t taddr = tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t(cbase + ch * 32);
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                    "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                    "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                      "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
                      "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
                      "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                    : "r"(taddr)
                    : "memory");
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (row < p.M) {
                    const int col0 = n0 + cbase + ch * 32;
                    float* yp = p.y + size_t(row) * p.N + col0;
                    // split K: every CTA adds into y (zeroed by the host unless the call accumulates); the residual rides
                    // with the first split
                    const float* rp = p.mode == 1 ? (split_k && blockIdx.z != 0 ? nullptr : p.residual + size_t(row) * p.N + col0)
                                                  : (p.mode == 2 && !split_k ? yp : nullptr);
#pragma unroll
                    for (int v = 0; v < 8; v++) {
                        if (col0 + v * 4 < p.N) {
                            float4 o = make_float4(__uint_as_float(r[4 * v]), __uint_as_float(r[4 * v + 1]),
                                                   __uint_as_float(r[4 * v + 2]), __uint_as_float(r[4 * v + 3]));
                            if (rp) {
                                const float4 a = __ldcg(reinterpret_cast<const float4*>(rp) + v);
                                o.x += a.x; o.y += a.y; o.z += a.z; o.w += a.w;
                            }
                            if (split_k)
                                asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(yp + 4 * v), "f"(o.x), "f"(o.y), "f"(o.z),
                                             "f"(o.w)
                                             : "memory");
                            else
                                reinterpret_cast<float4*>(yp)[v] = o;
                        }
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(uint32_t(kBN2)) : "memory");
    }
}

// ---------------------------------------------------------------------------------------------
// Calls of many rows: 256 x 256 output tiles, so that every dequantised weight feeds two 128-row MMAs.
// The 128-row kernel above is bound by the issue of the dequantisation (342 warp instructions per warp and 64-row stage
// against 512 tensor-pipe cycles); with 256 rows the same instructions stand against 1024 cycles, and the activations
// come by TMA instead of cp.async.  One CTA per SM: 512 TMEM columns (two 128 x 256 accumulators), three stages of 64 KB
// (2 x 16 KB activations, 32 KB weights).  Warps 0-15 dequantise and write results, warp 16 issues the MMAs, warp 17 the
// activation boxes.  The dequantising warps form two halves that fill alternate stages: with eight warps a stage took
// 1900 cycles, most of them waiting (for packed words, for the stage, for stores to become visible).  The weight tile is
// MN-major, so that a packed word becomes one 16-byte store without a transposition and a warp reads its words in
// 128-byte runs.
// Every CTA takes as many whole tiles as all CTAs can have.  What is left is dealt in units of one quantisation group (128
// weight rows) of one tile: an equal run of the units of the remaining full-height tiles and an equal run of those of the
// last, shorter tile row, so there is no partial wave whatever the shape.  Results leave through a 2 KB shared-memory patch per warp and TMA: a plain store where the run
// covered the whole contraction and y is to be overwritten, else an fp32 add-reduction.
constexpr int kTileM4 = 256, kTileN4 = 256, kStages4 = 3;
constexpr int kStageA4 = kTileM4 * kBK * 2, kStageB4 = kTileN4 * kBK * 2;  // 32 KB each
constexpr int kBlockB4 = kBK * 128;  // 64 weight rows of 64 columns
constexpr int kPatch4 = 32 * 16 * 4;
constexpr int kHalfThreads4 = 256;                // the warps that fill one stage; two such halves take turns
constexpr int kThreads4 = 2 * kHalfThreads4 + 64;
constexpr size_t kSmem4 = 1024 + size_t(kStages4) * (kStageA4 + kStageB4) + 16 * kPatch4;

struct GemmCall4 {
    CUtensorMap x_map;      // fp16 activations [M, K], box 64 x 128 rows, 128-byte swizzle
    CUtensorMap y_map;      // y [M, N], box 16 columns x 32 rows, 64-byte swizzle
    const uint32_t* qw;
    const uint32_t* qz;
    const __half* scales;
    const float* residual;  // rides with the first group of a tile
    int M, K, N;
    int add;                // 1: y already holds the addend (or zeros): every result is added
    int m_tiles, n_tiles, groups;
    int whole_tiles;           // tiles that a CTA has to itself; they come first
    int full_units, full_run;  // end of the units of the tile rows of 256 rows; units of them per CTA behind the whole tiles
    int tail_units, tail_run;  // the same for a last tile row of fewer rows
    int spins;                 // polls after which a wait gives up
    int drop;                  // test aid: the activations of this stage use of every CTA are never fetched (-1: none)
};

__global__ void __launch_bounds__(kThreads4, 1) awq_gemm_tc4_kernel(const __grid_constant__ GemmCall4 p) {
    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem = (smem_addr(smem_raw) + 1023u) & ~1023u;
    const uint32_t sA = smem, sB = smem + kStages4 * kStageA4, sY = sB + kStages4 * kStageB4;
    __shared__ uint64_t full_bar[kStages4], free_bar[kStages4], tile_bar, drained_bar, exit_bar;
    __shared__ uint32_t s_tmem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < kStages4; i++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&full_bar[i])), "r"(uint32_t(kHalfThreads4 / 32 + 1)));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&free_bar[i])));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&drained_bar)), "r"(uint32_t(2 * kHalfThreads4 / 32)));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&tile_bar)));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&exit_bar)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    pdl_launch_dependents();

    // ---- this CTA's units: whole tiles, a run of the other full tile rows, a run of the last tile row.  Unit u of the full
    // rows is group u % groups of tile u / groups, whose row index runs fastest (neighbouring CTAs share weights)
    const int full_rows = p.m_tiles - (p.tail_units > 0 ? 1 : 0);
    const int n_whole = p.whole_tiles * p.groups, w0 = int(blockIdx.x) * n_whole;
    const int f0 = min(int(gridDim.x) * n_whole + int(blockIdx.x) * p.full_run, p.full_units), f1 = min(f0 + p.full_run, p.full_units);
    const int n_full = n_whole + f1 - f0;
    // the tail is dealt from the last CTA down: it evens out the run that the last CTAs have less of
    const int rb = int(gridDim.x) - 1 - int(blockIdx.x);
    const int t0 = min(rb * p.tail_run, p.tail_units), t1 = min(t0 + p.tail_run, p.tail_units);
    const int n_units = n_full + t1 - t0;
    struct Unit { int mt, nt, group; };
    auto unit_at = [&](int i) {
        Unit r;
        if (i < n_full) {
            const int u = i < n_whole ? w0 + i : f0 + i - n_whole, tile = u / p.groups;
            r.group = u - tile * p.groups;
            r.nt = tile / full_rows;
            r.mt = tile - r.nt * full_rows;
        } else {
            const int u = t0 + i - n_full;
            r.nt = u / p.groups;
            r.group = u - r.nt * p.groups;
            r.mt = full_rows;
        }
        return r;
    };
    auto unit_after = [&](int i, const Unit& u) {  // unit i + 1, where unit i is u
        if (u.group + 1 == p.groups || i + 1 == n_full) return unit_at(i + 1);
        return Unit{u.mt, u.nt, u.group + 1};
    };
    // the run leaves a tile after unit i
    auto tile_ends = [&](int i, int group) { return group + 1 == p.groups || i + 1 == n_units || i + 1 == n_full; };

    if (warp == 17) {
        // ------------------------------------------------------------ activations
        if (lane == 0) {
            pdl_wait();
            bool dead = false;
            int it = 0;
            Unit u = {0, 0, 0};
            for (int i = 0; i < n_units && !dead; i++) {
                u = i == 0 ? unit_at(0) : unit_after(i - 1, u);
                const int boxes = p.M - u.mt * kTileM4 > kBM ? 2 : 1;
                for (int h = 0; h < 2; h++, it++) {
                    const int s = it % kStages4;
                    if (it >= kStages4 && !tc_mbar_wait(&free_bar[s], uint32_t(it / kStages4 - 1) & 1u, p.spins)) {
                        atomicExch(&g_gemm_wait_error, 21);
                        dead = true;
                        break;
                    }
                    if (it == p.drop) continue;
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&full_bar[s])),
                                 "r"(uint32_t(boxes * kStageA2))
                                 : "memory");
                    for (int b = 0; b < boxes; b++)
                        asm volatile(
                            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                            ::"r"(sA + s * kStageA4 + b * kStageA2), "l"(&p.x_map), "r"(u.group * 128 + h * kBK),
                            "r"(u.mt * kTileM4 + b * kBM), "r"(smem_addr(&full_bar[s]))
                            : "memory");
                }
            }
            // the copies in flight have to land before the block may end, whoever's wait ran out (otherwise this costs nothing)
            for (int j = it - kStages4 < 0 ? 0 : it - kStages4; j < it; j++)
                tc_mbar_wait(&full_bar[j % kStages4], uint32_t(j / kStages4) & 1u, p.spins);
        }
    } else if (warp == 16) {
        // ------------------------------------------------------------ MMA issue
        if (lane == 0) {
            const uint32_t idesc = (1u << 4) | (1u << 16) | (uint32_t(kTileN4 >> 3) << 17) | (uint32_t(kBM >> 4) << 24);  // B is MN-major
            bool dead = false, fresh = true;  // fresh: the next MMA starts a tile
            int it = 0, tiles = 0;
            Unit u = {0, 0, 0};
            for (int i = 0; i < n_units && !dead; i++) {
                u = i == 0 ? unit_at(0) : unit_after(i - 1, u);
                const int halves = p.M - u.mt * kTileM4 > kBM ? 2 : 1;
                // a new tile overwrites the accumulators: every warp has to have read the last one's
                if (fresh && tiles > 0 && !tc_mbar_wait(&drained_bar, uint32_t(tiles - 1) & 1u, p.spins)) {
                    atomicExch(&g_gemm_wait_error, 25);
                    break;
                }
                for (int h = 0; h < 2; h++, it++) {
                    const int s = it % kStages4;
                    if (!tc_mbar_wait(&full_bar[s], uint32_t(it / kStages4) & 1u, p.spins)) {
                        atomicExch(&g_gemm_wait_error, 22);
                        dead = true;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    for (int m = 0; m < halves; m++) {
#pragma unroll
                        for (int kk = 0; kk < kBK / 16; kk++) {
                            const uint64_t adesc = make_desc(sA + s * kStageA4 + m * kStageA2 + kk * 32);
                            const uint64_t bdesc = make_desc(sB + s * kStageB4 + kk * 2048) | (uint64_t(kBlockB4 >> 4) << 16);
                            const uint32_t accumulate = (fresh && kk == 0) ? 0u : 1u;
                            asm volatile(
                                "{\n\t.reg .pred p;\n\t"
                                "setp.ne.b32 p, %4, 0;\n\t"
                                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                                ::"r"(tmem + m * kTileN4), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
                                : "memory");
                        }
                    }
                    fresh = false;
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(&free_bar[s]))
                                 : "memory");
                }
                if (tile_ends(i, u.group)) {
                    fresh = true;
                    tiles++;
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(&tile_bar))
                                 : "memory");
                }
            }
            // every MMA issued is done before the block gives its tensor memory back, whoever's wait ran out (otherwise the
            // results have waited for them)
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(&exit_bar)) : "memory");
            tc_mbar_wait(&exit_bar, 0, p.spins);
        }
    } else {
        // ------------------------------------------------------------ dequantisation and results
        const int NW = p.N >> 3;
        const int half = warp >> 3;                                // fills the stages 2 i + half
        const int koct = warp & 7, j = lane;  // eight weight rows of packed word column j: a warp reads 128-byte runs
        auto load_w = [&](const Unit& u, uint32_t (&w)[8]) {
            const int wcol = u.nt * (kTileN4 / 8) + j;
            const bool ok = wcol < NW;
            const uint32_t* src = p.qw + size_t(u.group * 128 + half * kBK + koct * 8) * NW + (ok ? wcol : 0);
#pragma unroll
            for (int r = 0; r < 8; r++) w[r] = ok ? __ldg(src + size_t(r) * NW) : 0u;
        };
        auto load_consts = [&](const Unit& u, uint32_t& zw, uint4& sraw) {
            const int wcol = u.nt * (kTileN4 / 8) + j;
            const bool ok = wcol < NW;
            zw = ok ? __ldg(p.qz + size_t(u.group) * NW + wcol) : 0u;
            sraw = ok ? __ldg(reinterpret_cast<const uint4*>(p.scales + size_t(u.group) * p.N) + wcol) : make_uint4(0, 0, 0, 0);
        };
        // a word's eight columns are a 16-byte chunk of its row: column block j / 8, chunk (j % 8) ^ (row % 8)
        uint32_t b_off[8];
#pragma unroll
        for (int r = 0; r < 8; r++) b_off[r] = uint32_t((j >> 3) * kBlockB4 + (koct * 8 + r) * 128 + (((j & 7) ^ r) << 4));
        bool dead = false;
        TileConsts tc;
        auto stage_step = [&](int it, const uint32_t (&w)[8]) {
            const int s = it % kStages4;
            if (it >= kStages4 && !dead && !tc_mbar_wait(&free_bar[s], uint32_t(it / kStages4 - 1) & 1u, p.spins)) {
                atomicExch(&g_gemm_wait_error, 23);
                dead = true;
            }
            if (dead) return;  // an arrival out of turn could complete a phase that a copy still belongs to
            const uint32_t dst = sB + s * kStageB4;
#pragma unroll
            for (int r = 0; r < 8; r++) {
                uint32_t d[4];
                dequant_word_consts(w[r], tc, d);
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + b_off[r]), "r"(d[0]), "r"(d[1]), "r"(d[2]), "r"(d[3]) : "memory");
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&full_bar[s])) : "memory");
        };

        uint32_t w[8], zw = 0;
        uint4 sraw = make_uint4(0, 0, 0, 0);
        Unit next = {0, 0, 0};
        if (n_units > 0) {
            next = unit_at(0);
            load_w(next, w);
            load_consts(next, zw, sraw);
        }
        int first_group = next.group;  // group at which the run entered the current tile
        bool waited = false;
        int tiles = 0;
        for (int i = 0; i < n_units; i++) {
            const Unit u = next;
            const bool more = i + 1 < n_units;
            if (more) next = unit_after(i, u);
            tc = make_tile_consts(zw, sraw);
            if (more) load_consts(next, zw, sraw);
            stage_step(2 * i + half, w);
            if (more) load_w(next, w);
            if (!tile_ends(i, u.group)) continue;

            // ---- results: every MMA of the tile is done (a barrier of its own: a half sees only every other phase of free_bar)
            if (!dead && !tc_mbar_wait(&tile_bar, uint32_t(tiles++) & 1u, p.spins)) {
                atomicExch(&g_gemm_wait_error, 24);
                dead = true;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (!waited) {
                pdl_wait();  // y (and the residual) belong to the preceding kernels until here
                waited = true;
            }
            const bool whole = first_group == 0 && u.group + 1 == p.groups;
            const bool add = p.add || !whole;
            // two accumulators: one per half; one accumulator: each half takes half of the columns
            const bool both = p.M - u.mt * kTileM4 > kBM;
            const int m = both ? half : 0, chunks = both ? 8 : 4, c0 = both ? 0 : half * 4;
            if (!dead) {
#pragma unroll 1
                for (int c = 0; c < chunks; c++) {
                    const int row0 = u.mt * kTileM4 + m * kBM + (warp & 3) * 32;
                    const int tcol = ((warp >> 2) & 1) * 128 + (c0 + c) * 16, col0 = u.nt * kTileN4 + tcol;
                    if (row0 >= p.M || col0 >= p.N) break;
                    uint32_t r[16];
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                        : "r"(tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t(m * kTileN4 + tcol))
                        : "memory");
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (p.residual && first_group == 0 && row0 + lane < p.M) {
                        const float* rp = p.residual + size_t(row0 + lane) * p.N + col0;
#pragma unroll
                        for (int v = 0; v < 4; v++)
                            if (col0 + v * 4 < p.N) {
                                const float4 a = __ldcg(reinterpret_cast<const float4*>(rp) + v);
                                r[4 * v] = __float_as_uint(__uint_as_float(r[4 * v]) + a.x);
                                r[4 * v + 1] = __float_as_uint(__uint_as_float(r[4 * v + 1]) + a.y);
                                r[4 * v + 2] = __float_as_uint(__uint_as_float(r[4 * v + 2]) + a.z);
                                r[4 * v + 3] = __float_as_uint(__uint_as_float(r[4 * v + 3]) + a.w);
                            }
                    }
                    // three patches in turn: the warp's own, and its share of the stage that its half fills next (no MMA
                    // reads a stage now); a patch is free once the box sent from it has been read
                    const uint32_t patch = c % 3 == 0 ? sY + warp * kPatch4
                                                      : sB + ((2 * i + 2 + half) % kStages4) * kStageB4 + ((warp & 7) * 2 + c % 3 - 1) * kPatch4;
                    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 2;" ::: "memory");
                    __syncwarp();
#pragma unroll
                    for (int v = 0; v < 4; v++)
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(patch + lane * 64 + ((v ^ ((lane >> 1) & 3)) << 4)), "r"(r[4 * v]),
                                     "r"(r[4 * v + 1]), "r"(r[4 * v + 2]), "r"(r[4 * v + 3])
                                     : "memory");
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        if (add)
                            asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.bulk_group [%0, {%1, %2}], [%3];" ::"l"(&p.y_map),
                                         "r"(col0), "r"(row0), "r"(patch)
                                         : "memory");
                        else
                            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(&p.y_map), "r"(col0),
                                         "r"(row0), "r"(patch)
                                         : "memory");
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            asm volatile("bar.sync %0, %1;" ::"r"(1 + half), "n"(kHalfThreads4) : "memory");  // the stage is the half's again
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&drained_bar)) : "memory");
            first_group = more ? next.group : 0;
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

using EncodeTiledTc = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledTc encode_fn_tc() {
    static EncodeTiledTc fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
        return reinterpret_cast<EncodeTiledTc>(f);
    }();
    return fn;
}
// row-major [rows, cols], boxes of box_cols (box_cols * elem_bytes = the swizzle's span) x box_rows, zero fill
bool encode_rows_map(CUtensorMap* out, CUtensorMapDataType type, int elem_bytes, const void* base, int rows, int cols, int box_cols, int box_rows,
                     CUtensorMapSwizzle swizzle) {
    EncodeTiledTc fn = encode_fn_tc();
    if (!fn) return false;
    const cuuint64_t dims[2] = {cuuint64_t(cols), cuuint64_t(rows)};
    const cuuint64_t strides[1] = {cuuint64_t(cols) * elem_bytes};
    const cuuint32_t box[2] = {cuuint32_t(box_cols), cuuint32_t(box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    return fn(out, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int g_gemm_tile_spins = kSpinLimitTc, g_gemm_tile_drop = -1;  // tuning keys "tile_wait_spins", "tile_drop_stage" (tests of the bounded waits)
int g_gemm_tile_always = 0;  // tuning key "gemm_tile_always": the tiles also where the other kernel is ahead (tests, measurements)
int g_gemm_tile_rows = 33;  // tuning key "gemm_tile_rows": fewest rows of a call that takes the 256 x 256 tiles; 0: none

// Whether a call takes the 256 x 256 tiles rather than the 128-row kernel.  They lead wherever the latter needs more than one wave of
// two CTAs per SM or finds nothing to split (4096 x 24576: 64 rows 37 against 45 us, 256 rows 50 / 85, 512 rows 96 / 165, 2048 rows
// 362 / 703), but for one case: between 257 and 511 rows they run a second, short tile row with its own unpacking and results, and the
// 128-row kernel is ahead where its K split happens to fill one wave (4096 x 6144, 300 rows: 34.0 against 38.1 us, 4096 x 2560 23.4 /
// 28.6; where it does not: 2560 x 6144 39.1 / 24.6).
// Where the split fits one wave, outputs of few tiles leave either kernel a chain of a few stages and a result of 128 or of 256
// rows to add.  There the estimates below decide; they were fitted to 1146 calls (33 to 2048 rows, K 384 to 9600, N 40 to 24 576) and are 9
// and 8 % off on average.  Taking the tiles for all of them cost up to 48 % (4096 x 744: 450 rows 17.0 us in the 128-row kernel, 25.1
// here; 384 x 232: 256 rows 9.1 / 12.4; 1024 x 6144: 700 rows 29.0 / 38.1; the other way round 4096 x 2560, 128 rows: 20.8 / 18.2).  A single
// group of K and a narrow output (128 x 40: 200 rows 5.7 / 7.1) is the one unsplit call that the 128-row kernel finishes first.
bool tiles_pay(int M, int K, int N, bool accumulate, int tiles128, int splits128) {
    const int ctas = tiles128 * splits128, sms = device_sm_count(), groups = K / 128;
    if (M > 256 && M < 512 && ctas * 2 >= sms * 3 && ctas <= 2 * sms) return false;
    if (splits128 == 1) return groups > 1 || N > 64 || accumulate;
    if (ctas > 2 * sms) return true;
    const float cols = float(N < 256 ? N : 256) / 256.f;
    // 128-row tiles, us: stages of a CTA (slower once CTAs share SMs), sums added by reductions, one result
    const float stages = float(2 * groups / splits128);
    const float rows_us = 2.46f + (ctas * 10 > sms * 7 ? 1.22f : 0.74f) * stages + 0.78f * float(ctas) / float(sms) +
                          0.96e-6f * float(M) * float(N) * float(splits128) + 3.92f * cols * float(M < 128 ? M : 128) / 128.f;
    // 256-row tiles, us: the busiest CTA's groups (two MMAs a stage, one in a last tile row of at most 128 rows) and results - a run whose
    // length does not divide a tile's groups may end in a second tile - and sums added by reductions.  A CTA may have a run of the full
    // tile rows, one of the last, or both.
    const int n_tiles = (N + kTileN4 - 1) / kTileN4, last = M % kTileM4;
    const int full = M / kTileM4 * n_tiles * groups, tail = last ? n_tiles * groups : 0;
    const int full_run = (full + sms - 1) / sms, tail_run = (tail + sms - 1) / sms;
    auto run_us = [&](int run, float group_us, float height) {
        const float results = run == 0 ? 0.f : (run > 1 && groups % run ? 2.f : 1.f);
        return group_us * float(run) + 5.74f * results * cols * height;
    };
    const float full_us = run_us(full_run, 1.77f, 1.f), tail_us = run_us(tail_run, last > 128 ? 1.77f : 1.45f, float(last) / kTileM4);
    const bool both = (full ? (full + full_run - 1) / full_run : 0) + (tail ? (tail + tail_run - 1) / tail_run : 0) > sms;
    const float adds = float(N) * 1e-6f * float(groups) *
                       ((full ? float(M - last) / float(full_run) : 0.f) + (tail ? float(last) / float(tail_run) : 0.f));
    const float tiles_us = 3.77f + (both ? full_us + tail_us : (full_us > tail_us ? full_us : tail_us)) + 0.31f * adds;
    return rows_us >= 0.93f * tiles_us;
}

// zeroes what a launch that overwrites y adds up from several CTAs: columns [col0, N) of every row and the rows from row0 on
__global__ void __launch_bounds__(256) zero_split_kernel(float4* y, int M, int N4, int row0, int col4) {
    pdl_launch_dependents();
    pdl_wait();
    const int m = blockIdx.x;
    for (int i = (m >= row0 ? 0 : col4) + threadIdx.x; i < N4; i += 256) y[size_t(m) * N4 + i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// y[add ? += : =] x16 . W (+ residual); share: tiles may be added up from several CTAs, otherwise every tile is one CTA's (a fixed
// order of the sums, at the price of a partial last wave)
int launch_tiles4(const GemmParams& g, const __half* x16, bool share, bool zeroed, cudaStream_t stream) {
    GemmCall4 c;
    memset(&c, 0, sizeof(c));
    if (!encode_rows_map(&c.x_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x16, g.M, g.K, kBK, kBM, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !encode_rows_map(&c.y_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, g.y, g.M, g.N, 16, 32, CU_TENSOR_MAP_SWIZZLE_64B)) {
        set_error("awq_gemm: tensor map encoding failed");
        return KUIPER_INTERNAL_ERROR;
    }
    c.qw = g.qw; c.qz = g.qz; c.scales = g.scales;
    c.residual = g.mode == 1 ? g.residual : nullptr;
    c.M = g.M; c.K = g.K; c.N = g.N;
    c.add = g.mode == 2;
    c.m_tiles = (g.M + kTileM4 - 1) / kTileM4;
    c.n_tiles = (g.N + kTileN4 - 1) / kTileN4;
    c.groups = g.K / 128;
    c.spins = g_gemm_tile_spins;
    c.drop = g_gemm_tile_drop;
    const int tail = g.M % kTileM4 != 0 ? 1 : 0, ctas = device_sm_count();
    c.full_units = (c.m_tiles - tail) * c.n_tiles * c.groups;
    c.tail_units = tail * c.n_tiles * c.groups;
    c.whole_tiles = (c.m_tiles - tail) * c.n_tiles / ctas;
    const int split_units = c.full_units - c.whole_tiles * ctas * c.groups;
    c.full_run = (split_units + ctas - 1) / ctas;
    c.tail_run = (c.tail_units + ctas - 1) / ctas;
    if (!share) {  // runs of whole tiles
        c.full_run = (c.full_run + c.groups - 1) / c.groups * c.groups;
        c.tail_run = (c.tail_run + c.groups - 1) / c.groups * c.groups;
    }
    static size_t configured[kMaxDevices] = {};
    if (!ensure_dynamic_smem(awq_gemm_tc4_kernel, kSmem4, configured)) {
        set_error("awq_gemm: cannot reserve %zu bytes of shared memory", kSmem4);
        return KUIPER_INTERNAL_ERROR;
    }
    if (!c.add && share && !zeroed && (split_units > 0 || tail)) {
        const int full_rows = c.m_tiles - tail;
        const int first_col = split_units > 0 ? c.whole_tiles * ctas / full_rows * kTileN4 : g.N;  // the first column tile that is not whole
        const int rc = pdl_status(launch_pdl(zero_split_kernel, dim3(g.M), dim3(256), 0, stream, reinterpret_cast<float4*>(g.y), g.M, g.N / 4,
                                             full_rows * kTileM4, first_col / 4),
                                  "awq_gemm zero");
        if (rc != KUIPER_OK) return rc;
    }
    return pdl_status(launch_pdl(awq_gemm_tc4_kernel, dim3(ctas), dim3(kThreads4), kSmem4, stream, c), "awq_gemm");
}

// Calls of up to 32 rows read the weights through the packed-word kernel of awq_gemm_rows.cu, one pass over them: 4096 x 24576
// (ten matrices in turn) 8 rows 13.8, 16 rows 16.7, 32 rows 29.6 us, where the 256 x 256 tiles take 38 us from one row to 64 (they
// are bound by the dequantisation there) and the 128-row tiles 46.
int g_gemm_rows_max = 32;  // tuning key "gemm_rows_max": most rows of such a call; 0 switches the path off

constexpr int kMaxSplitK = 8;
int g_gemm_split_k = 1;  // tuning key "gemm_split_k": 0 switches the K split of the third generation off
// tuning key "gemm_impl": 3 (as shipped) lets the rules above choose; 2 keeps every call on 128-row tiles handed over at a block-wide
// barrier (awq_gemm_tc2_kernel)
int g_gemm_impl = 3;

}  // namespace

int awq_rows_launch(const __half* x16, const int32_t* qweight, const int32_t* qzeros, const uint16_t* scales, float* y, const float* residual,
                    int M, int K, int N, cudaStream_t stream);
int awq_rows_status();
void awq_rows_set_tuning(const char* key, int value);

// x (n4 float4s) -> fp16; also zeroes zero4 float4s
int convert_f16_launch(const float* x, __half* out, int64_t n4, float* zero, int64_t zero4, cudaStream_t stream) {
    int blocks = int(((n4 > zero4 ? n4 : zero4) + 255) / 256);
    if (blocks > 148 * 8) blocks = 148 * 8;
    return pdl_status(launch_pdl(convert_f16_kernel, dim3(blocks), dim3(256), 0, stream, reinterpret_cast<const float4*>(x),
                                 reinterpret_cast<uint2*>(out), n4, reinterpret_cast<float4*>(zero), zero4),
                      "awq_gemm convert");
}

void awq_gemm_set_tuning(const char* key, int value) {
    if (!strcmp(key, "gemm_impl")) g_gemm_impl = value == 3 ? 3 : 2;
    if (!strcmp(key, "gemm_tile_rows")) g_gemm_tile_rows = value < 0 ? 0 : value;
    if (!strcmp(key, "gemm_tile_always")) g_gemm_tile_always = value != 0;
    if (!strcmp(key, "tile_wait_spins")) g_gemm_tile_spins = value < 1 ? kSpinLimitTc : value;
    if (!strcmp(key, "tile_drop_stage")) g_gemm_tile_drop = value;
    if (!strcmp(key, "gemm_rows_max")) g_gemm_rows_max = value < 0 ? 0 : value;
    awq_rows_set_tuning(key, value);
    if (!strcmp(key, "gemm_split_k")) g_gemm_split_k = value < 0 ? 0 : value;
}

}  // namespace kuiper

using namespace kuiper;

extern "C" int kuiper_awq_gemm_status(void) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_gemm_wait_error, sizeof(int)) != cudaSuccess) v = -1;
    if (v == 0) v = awq_rows_status();
    if (v == 0) return KUIPER_OK;
    set_error("awq_gemm: a bounded tensor-core pipeline wait ran out (code %d)", v);
    return KUIPER_INTERNAL_ERROR;
}

extern "C" size_t kuiper_awq_gemm_workspace_bytes(int M, int K) {
    if (M <= 0 || K <= 0) return 0;
    return (size_t(M) * size_t(K) * sizeof(__half) + 255) / 256 * 256;  // fp16 copy of the activations
}

// Shared by the entry points: x is fp32 (converted into the workspace first) or already fp16 (x16, no workspace).
static int gemm_common(const float* x, const __half* x16_in, const int32_t* qweight, const int32_t* qzeros, const uint16_t* scales,
                       float* y, const float* residual, int accumulate, bool any_order, int M, int K, int N, int group,
                       void* workspace, size_t workspace_bytes, kuiper_stream_t stream) {
    KUIPER_REQUIRE((x || x16_in) && qweight && qzeros && scales && y, "awq_gemm: null tensor pointer");
    KUIPER_REQUIRE(M > 0 && K > 0 && N > 0, "awq_gemm: empty shape M=%d K=%d N=%d", M, K, N);
    KUIPER_REQUIRE(group == 128, "awq_gemm: group size %d is not supported (128 only)", group);
    KUIPER_REQUIRE(K % 128 == 0 && N % 8 == 0, "awq_gemm: needs K %% 128 == 0 and N %% 8 == 0 (K=%d N=%d)", K, N);
    KUIPER_REQUIRE(!(accumulate && residual), "awq_gemm: accumulate and residual are exclusive");
    KUIPER_REQUIRE(((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(x16_in) | reinterpret_cast<uintptr_t>(y) |
                     reinterpret_cast<uintptr_t>(scales) | reinterpret_cast<uintptr_t>(residual)) & 15) == 0 && (N % 4 == 0),
                   "awq_gemm: x, y, scales and residual must be 16-byte aligned");
    GemmParams p;
    p.x = x;
    p.qw = reinterpret_cast<const uint32_t*>(qweight);
    p.qz = reinterpret_cast<const uint32_t*>(qzeros);
    p.scales = reinterpret_cast<const __half*>(scales);
    p.y = y;
    p.residual = residual;
    p.M = M; p.K = K; p.N = N;
    p.mode = accumulate ? 2 : (residual ? (residual == y ? 2 : 1) : 0);  // y + residual with residual == y is y += 
    KUIPER_REQUIRE(x16_in != nullptr || (workspace != nullptr && workspace_bytes >= kuiper_awq_gemm_workspace_bytes(M, K) &&
                                         (reinterpret_cast<uintptr_t>(workspace) & 15) == 0),
                   "awq_gemm: needs a 16-byte aligned workspace of kuiper_awq_gemm_workspace_bytes(M, K) bytes (got %zu)",
                   workspace_bytes);
    const int64_t n4 = x16_in ? 0 : int64_t(M) * K / 4;  // activations that arrive as fp16 need no conversion
    __half* const x16_ws = reinterpret_cast<__half*>(workspace);
    const bool few_rows = g_gemm_impl == 3 && g_gemm_split_k == 1 && M <= g_gemm_rows_max && N % 32 == 0 &&
                          ((reinterpret_cast<uintptr_t>(qweight) | reinterpret_cast<uintptr_t>(qzeros)) & 15) == 0;
    if (few_rows) {
        const int64_t zero4 = p.mode != 2 ? int64_t(M) * N / 4 : 0;
        if (n4 > 0 || zero4 > 0) {
            const int rc = convert_f16_launch(x, x16_ws, n4, y, zero4, as_stream(stream));
            if (rc != KUIPER_OK) return rc;
        }
        return awq_rows_launch(x16_in ? x16_in : x16_ws, qweight, qzeros, scales, y, p.mode == 1 ? residual : nullptr, M, K, N, as_stream(stream));
    }
    // Few output tiles (a decode batch, a short chunk: one row of tiles is N / 256 CTAs) leave most SMs without work while
    // every CTA streams a whole column panel of the weight: the third generation then splits K so that about two CTAs
    // per SM are busy.  A split is a whole number of 128-row groups; the sums meet through reductions, so y starts from
    // zero (or from its content when the call accumulates) and the summation order is no longer fixed.
    const dim3 grid2((N + kBN2 - 1) / kBN2, (M + kBM - 1) / kBM, 1);
    int splits = 1;
    if (g_gemm_impl == 3 && g_gemm_split_k) {
        // up to a third of a second wave is still a gain (measured: 96 tiles run 48 us with 4 splits, 55 us with 2)
        const int tiles = int(grid2.x * grid2.y), groups = K / 128, want = (2 * device_sm_count() * 4 / 3 + tiles - 1) / tiles;
        for (int sdiv = 2; sdiv <= groups && sdiv <= kMaxSplitK && sdiv <= want; sdiv++)
            if (groups % sdiv == 0) splits = sdiv;
        if (g_gemm_split_k > 1 && groups % g_gemm_split_k == 0) splits = g_gemm_split_k;  // forced (measurement aid)
    }
    if (g_gemm_impl == 3 && g_gemm_split_k == 1 && g_gemm_tile_rows > 0 && M >= g_gemm_tile_rows && encode_fn_tc() != nullptr &&
        (g_gemm_tile_always || tiles_pay(M, K, N, p.mode == 2, int(grid2.x * grid2.y), splits))) {
        const bool share = any_order || splits > 1;
        // where no tile is whole, the launch that converts the activations zeroes y as well
        const bool zero_all = share && n4 > 0 && p.mode != 2 && (M / kTileM4) * ((N + kTileN4 - 1) / kTileN4) < device_sm_count();
        if (n4 > 0) {
            const int rc = convert_f16_launch(x, x16_ws, n4, y, zero_all ? int64_t(M) * N / 4 : 0, as_stream(stream));
            if (rc != KUIPER_OK) return rc;
        }
        return launch_tiles4(p, x16_in ? x16_in : x16_ws, share, zero_all, as_stream(stream));
    }
    const bool zero_y = splits > 1 && p.mode != 2;
    // activations converted to fp16 once (the same launch zeroes y for a split call), then 128 x 256 output tiles
    const int64_t zero4 = zero_y ? int64_t(M) * N / 4 : 0;
    if (n4 > 0 || zero4 > 0) {
        const int rc = convert_f16_launch(x, x16_ws, n4, y, zero4, as_stream(stream));
        if (rc != KUIPER_OK) return rc;
    }
    GemmParams2 p2;
    p2.g = p;
    p2.x16 = x16_in ? x16_in : x16_ws;
    p2.tiles_per_split = 0;
    const size_t smem2 = 1024 + size_t(kStages2) * (kStageA2 + kStageB2);
    if (g_gemm_impl == 3) {
        static size_t configured3[kMaxDevices] = {};
        if (!ensure_dynamic_smem(awq_gemm_tc3_kernel, smem2, configured3)) {
            set_error("awq_gemm: cannot reserve %zu bytes of shared memory", smem2);
            return KUIPER_INTERNAL_ERROR;
        }
        dim3 grid3 = grid2;
        if (splits > 1) {
            grid3.z = splits;
            p2.tiles_per_split = (K / kBK) / splits;
        }
        return pdl_status(launch_pdl(awq_gemm_tc3_kernel, grid3, dim3(kGemmThreads3), smem2, as_stream(stream), p2), "awq_gemm");
    }
    static size_t configured[kMaxDevices] = {};
    if (!ensure_dynamic_smem(awq_gemm_tc2_kernel, smem2, configured)) {
        set_error("awq_gemm: cannot reserve %zu bytes of shared memory", smem2);
        return KUIPER_INTERNAL_ERROR;
    }
    return pdl_status(launch_pdl(awq_gemm_tc2_kernel, grid2, dim3(kGemmThreads), smem2, as_stream(stream), p2), "awq_gemm");
}

extern "C" int kuiper_awq_gemm_f32(const float* x, const int32_t* qweight, const int32_t* qzeros, const uint16_t* scales,
                                   float* y, const float* residual, int accumulate, int M, int K, int N, int group,
                                   void* workspace, size_t workspace_bytes, kuiper_stream_t stream) {
    KUIPER_REQUIRE(x != nullptr, "awq_gemm: null tensor pointer");
    return gemm_common(x, nullptr, qweight, qzeros, scales, y, residual, accumulate, false, M, K, N, group, workspace, workspace_bytes, stream);
}

extern "C" int kuiper_awq_gemm_f16in_f32(const uint16_t* x16, const int32_t* qweight, const int32_t* qzeros, const uint16_t* scales,
                                         float* y, const float* residual, int accumulate, int M, int K, int N, int group,
                                         kuiper_stream_t stream) {
    KUIPER_REQUIRE(x16 != nullptr, "awq_gemm_f16in: null tensor pointer");
    return gemm_common(nullptr, reinterpret_cast<const __half*>(x16), qweight, qzeros, scales, y, residual, accumulate, false, M, K, N, group,
                       nullptr, 0, stream);
}

extern "C" int kuiper_awq_gemm_any_order_f32(const float* x, const uint16_t* x16, const int32_t* qweight, const int32_t* qzeros,
                                             const uint16_t* scales, float* y, const float* residual, int accumulate, int M, int K, int N,
                                             int group, void* workspace, size_t workspace_bytes, kuiper_stream_t stream) {
    KUIPER_REQUIRE((x != nullptr) != (x16 != nullptr), "awq_gemm_any_order: exactly one of x and x16 is given");
    return gemm_common(x, reinterpret_cast<const __half*>(x16), qweight, qzeros, scales, y, residual, accumulate, true, M, K, N, group,
                       workspace, workspace_bytes, stream);
}

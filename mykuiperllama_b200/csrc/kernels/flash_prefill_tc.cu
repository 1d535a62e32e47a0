// Causal attention of a prompt chunk on the 5th-generation tensor cores (tcgen05, accumulators and probabilities in tensor
// memory); same operation, operands and precision as flash_prefill.cu, which keeps the short chunks.
// Placeholder it fills: kuiper/include/op/mha.h:1-11 of the reference.
//
// The work is a contraction: with q and the probabilities as bf16 high + low parts (16 significant bits, K and V are
// exact bf16) it takes four products of 128 x 128 x 128 per 128 query vectors and 128 cache rows.  The scheme is the one published
// for FlashAttention-4: two query tiles in turn, probabilities over their scores in tensor memory, a running maximum that
// moves only past a factor.  A CTA owns one kv head
// and 256 query vectors (row, head) = two query tiles of 128; while one tile's softmax runs, the tensor cores work for the
// other.
//   S_w = Q_w . K^T   A = q parts in shared memory (K-major, 128-byte swizzle), B = K tile as TMA lays it down
//   softmax           four warps per query tile, one vector per thread; the running maximum moves (and O is rescaled)
//                     only where it has grown by more than a factor 2^8, which changes no result: every probability and
//                     the row sum refer to the same maximum
//   O_w += P_w . V    A = probability parts in tensor memory (over the scores they came from), B = V tile, MN-major
// K and V tiles of 128 rows alternate through a ring of three 32 KB slots.  Cache rows past the chunk's end read as zeros
// (the tensor maps end there), so nothing beyond the written rows is ever multiplied.  A hidden row's probability is 0, and 0
// times a V that is not finite is NaN, so the second product stops at the 16 rows that hold the last one visible to any vector
// of its query tile (128 / R token rows; the tiled kernel stops at a multiple of 64).
// Tensor memory: two tiles x (128 columns S / P + 128 columns O) = all 512 columns; one CTA per SM, longest rows first.
// Every mbarrier wait is bounded; on a timeout an error word is recorded, the block stops and frees its tensor memory.
#include <cuda.h>
#include <cstring>

#include "common.cuh"

namespace kuiper {
namespace {

constexpr int kTD = 128;                        // head dimension
constexpr int kTRows = 128;                     // cache rows of a tile
constexpr int kTSlot = kTRows * kTD * 2;        // 32 KB: two 64-dimension halves of 128 rows x 128 bytes
constexpr int kTSlots = 3;
constexpr int kTQ = 2 * kTSlot;                 // high and low parts of one query tile
constexpr int kTThreads = 256 + 64;             // two softmax warpgroups, MMA warp, load warp
constexpr size_t kTSmem = 1024 + 2 * kTQ + kTSlots * kTSlot;
constexpr int kTSpin = 1 << 22;  // polls of one wait, about a microsecond each

__device__ int g_prefill_wait_error = 0;

struct PrefillTcCall {
    CUtensorMap k_map, v_map;  // [heads][pos0 + M][128] bf16, box 64 x 128 x 1
    const float* q;            // [M, Nq, 128]
    float* out;
    int M, Nq, Nkv, pos0, head0;  // head0: first head of the sequence's slot in the cache
    int R;
    int spins;  // polls after which a wait gives up
    int drop;   // test aid: this K or V tile (in the order K0 V0 K1 V1 ...) is never fetched (-1: none)
};

__device__ __forceinline__ uint32_t ts_u32(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ bool ts_wait(uint64_t* bar, uint32_t parity, int spins) {
    const uint32_t addr = ts_u32(bar);
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
__device__ __forceinline__ void ts_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(ts_u32(bar)) : "memory");
}
__device__ __forceinline__ void ts_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(ts_u32(bar)) : "memory");
}
// 128-byte swizzle descriptors: K-major operands step 1024 B per eight rows; the MN-major V tile steps 1024 B per eight
// cache rows (stride) and 16 KB per 64 dimensions (leading)
__device__ __forceinline__ uint64_t ts_desc(uint32_t saddr, uint32_t leading) {
    return uint64_t((saddr >> 4) & 0x3fffu) | (uint64_t((leading >> 4) & 0x3fffu) << 16) | (uint64_t(1024u >> 4) << 32) | (uint64_t(1) << 46) |
           (uint64_t(2) << 61);
}
__device__ __forceinline__ void ts_ld32(uint32_t taddr, float* v) {
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void ts_st32(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]),
        "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
// (x, y) as bf16 high parts in one register (x in the low half) and what is left of them as bf16 low parts
__device__ __forceinline__ void ts_split(float x, float y, uint32_t& hi, uint32_t& lo) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(y), "f"(x));
    const float xr = x - __uint_as_float(hi << 16), yr = y - __uint_as_float(hi & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(yr), "f"(xr));
}

__global__ void __launch_bounds__(kTThreads, 1) flash_prefill_tc_kernel(const __grid_constant__ PrefillTcCall p) {
    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem = (ts_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t sQ = smem, sKV = smem + 2 * kTQ;
    __shared__ uint64_t slot_full[kTSlots], slot_free[kTSlots], s_ready[2], p_ready[2], o_ready[2], q_ready, exit_bar;
    __shared__ uint32_t s_tmem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        auto init = [](uint64_t* bar, uint32_t count) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(ts_u32(bar)), "r"(count));
        };
        for (int i = 0; i < kTSlots; i++) {
            init(&slot_full[i], 1);
            init(&slot_free[i], 1);
        }
        for (int w = 0; w < 2; w++) {
            init(&s_ready[w], 1);
            init(&p_ready[w], 4);
            init(&o_ready[w], 1);
        }
        init(&q_ready, 8);
        init(&exit_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ts_u32(&s_tmem)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    pdl_launch_dependents();

    const int kvh = blockIdx.y;
    const int block = int(gridDim.x) - 1 - int(blockIdx.x);  // the blocks with the most cache rows start first
    const int vec0 = block * 256;                            // first (row, head) vector of this block
    const int n_vec = p.M * p.R;
    const int last_row = min(vec0 + 255, n_vec - 1) / p.R;
    const int n_tiles = (p.pos0 + last_row + kTRows) / kTRows;

    if (warp == 9) {
        // ------------------------------------------------------------ K and V tiles
        if (lane == 0) {
            pdl_wait();  // the newest cache rows come from the preceding kernel
            int i = 0;
            for (; i < 2 * n_tiles; i++) {  // K0 V0 K1 V1 ...
                const int s = i % kTSlots;
                if (i >= kTSlots && !ts_wait(&slot_free[s], uint32_t(i / kTSlots - 1) & 1u, p.spins)) {
                    atomicExch(&g_prefill_wait_error, 31);
                    break;
                }
                if (i == p.drop) continue;
                const CUtensorMap* map = (i & 1) ? &p.v_map : &p.k_map;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(ts_u32(&slot_full[s])), "r"(uint32_t(kTSlot)) : "memory");
                for (int h = 0; h < 2; h++)
                    asm volatile(
                        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                        ::"r"(sKV + s * kTSlot + h * (kTSlot / 2)), "l"(map), "r"(h * 64), "r"((i >> 1) * kTRows), "r"(p.head0 + kvh),
                        "r"(ts_u32(&slot_full[s]))
                        : "memory");
            }
            // the copies in flight have to land before the block may end, whoever's wait ran out (otherwise this costs nothing)
            for (int j = max(i - kTSlots, 0); j < i; j++) ts_wait(&slot_full[j % kTSlots], uint32_t(j / kTSlots) & 1u, p.spins);
        }
    } else if (warp == 8) {
        // ------------------------------------------------------------ MMA issue
        if (lane == 0) {
            // fp32 accumulator, bf16 operands, M = N = 128; the second one has an MN-major B
            const uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(128 >> 3) << 17) | (uint32_t(128 >> 4) << 24);
            const uint32_t idesc_o = idesc_s | (1u << 16);
            bool dead = false;
            auto need = [&](uint64_t* bar, uint32_t parity) {
                if (dead || ts_wait(bar, parity, p.spins)) return;
                atomicExch(&g_prefill_wait_error, 32);
                dead = true;
            };
            auto scores = [&](int w, int j) {  // S_w = Q_w . K_j^T
                const int s = (2 * j) % kTSlots;
                need(&slot_full[s], uint32_t(2 * j / kTSlots) & 1u);
                if (dead) return;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int part = 1; part >= 0; part--)  // the low parts first: the accumulator truncates, and they add while it is small
#pragma unroll
                    for (int kk = 0; kk < 8; kk++) {
                        const uint32_t off = (kk >> 2) * (kTSlot / 2) + (kk & 3) * 32;
                        const uint64_t a = ts_desc(sQ + w * kTQ + part * kTSlot + off, 0), b = ts_desc(sKV + s * kTSlot + off, 0);
                        const uint32_t acc = (part == 0 || kk) ? 1u : 0u;
                        asm volatile(
                            "{\n\t.reg .pred p;\n\t"
                            "setp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                            ::"r"(tmem + w * 256), "l"(a), "l"(b), "r"(idesc_s), "r"(acc)
                            : "memory");
                    }
                ts_commit(&s_ready[w]);
                if (w == 1) ts_commit(&slot_free[s]);
            };
            // last cache row that any vector of each query tile sees
            const int last0 = p.pos0 + min(vec0 + 127, n_vec - 1) / p.R, last1 = p.pos0 + last_row;
            need(&q_ready, 0);
            scores(0, 0);
            scores(1, 0);
            for (int j = 0; j < n_tiles && !dead; j++)
                for (int w = 0; w < 2 && !dead; w++) {
                    const int s = (2 * j + 1) % kTSlots;
                    const int seen = (w == 0 ? last0 : last1) - j * kTRows;  // last row of this tile that w sees
                    need(&slot_full[s], uint32_t((2 * j + 1) / kTSlots) & 1u);
                    need(&p_ready[w], uint32_t(j) & 1u);
                    if (dead) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    // O_w += P_w . V_j; per 32 cache rows: 16 columns of high parts, 16 of low parts
                    auto product = [&](int kk) {
#pragma unroll
                        for (int part = 0; part < 2; part++) {
                            const uint32_t a = tmem + w * 256 + (kk >> 1) * 32 + part * 16 + (kk & 1) * 8;
                            const uint64_t b = ts_desc(sKV + s * kTSlot + kk * 2048, kTSlot / 2);
                            const uint32_t acc = (j | part | kk) ? 1u : 0u;
                            asm volatile(
                                "{\n\t.reg .pred p;\n\t"
                                "setp.ne.b32 p, %4, 0;\n\t"
                                "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                                ::"r"(tmem + w * 256 + 128), "r"(a), "l"(b), "r"(idesc_o), "r"(acc)
                                : "memory");
                        }
                    };
                    // (whole tiles apart: 2048 rows of 32 / 8 heads 102.3 us, as without a bound; one loop with the bound for all 104.3)
                    if (seen >= kTRows - 16) {
#pragma unroll
                        for (int kk = 0; kk < 8; kk++) product(kk);
                    } else {
#pragma unroll 1
                        for (int kk = 0; kk * 16 <= seen; kk++) product(kk);
                    }
                    if (w == 1) ts_commit(&slot_free[s]);
                    if (j + 1 == n_tiles)
                        ts_commit(&o_ready[w]);
                    else
                        scores(w, j + 1);  // its commit also says that O_w is complete up to tile j
                }
            // every MMA issued is done before the block gives its tensor memory back, whoever's wait ran out
            ts_commit(&exit_bar);
            ts_wait(&exit_bar, 0, p.spins);
        }
    } else {
        // ------------------------------------------------------------ softmax: thread = one query vector
        const int w = warp >> 2, row = tid & 127;
        const int vec = vec0 + w * 128 + row;
        auto vector_at = [&](int v) {  // offset of a vector in q and out; those past the end stand in for the last one
            v = min(v, n_vec - 1);
            return (size_t(v / p.R) * p.Nq + kvh * p.R + v % p.R) * kTD;
        };
        const int m = min(vec, n_vec - 1) / p.R;
        const int last = p.pos0 + m;  // last visible cache row
        pdl_wait();
        {
            // a warp writes its 32 vectors one after another, a lane four dimensions of each (whole 512-byte rows are read)
            const float scale = 0.08838834764831845f;
            const uint32_t dst0 = sQ + w * kTQ + (lane >> 4) * (kTSlot / 2) + (lane & 1) * 8;
#pragma unroll 8
            for (int i = 0; i < 32; i++) {
                const int r = (warp & 3) * 32 + i;
                const float4 x = __ldcg(reinterpret_cast<const float4*>(p.q + vector_at(vec0 + w * 128 + r)) + lane);
                uint32_t hi[2], lo[2];
                ts_split(x.x * scale, x.y * scale, hi[0], lo[0]);
                ts_split(x.z * scale, x.w * scale, hi[1], lo[1]);
                const uint32_t dst = dst0 + r * 128 + ((((lane >> 1) & 7) ^ (r & 7)) << 4);
                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst), "r"(hi[0]), "r"(hi[1]) : "memory");
                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst + kTSlot), "r"(lo[0]), "r"(lo[1]) : "memory");
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) ts_arrive(&q_ready);
        }
        const uint32_t lanes = uint32_t((warp & 3) * 32) << 16;
        const uint32_t tS = tmem + lanes + w * 256, tO = tS + 128;
        constexpr float kLog2e = 1.4426950408889634f;
        float mx = -INFINITY, sum = 0.f;
        bool dead = false;
        for (int j = 0; j < n_tiles; j++) {
            if (!ts_wait(&s_ready[w], uint32_t(j) & 1u, p.spins)) {
                atomicExch(&g_prefill_wait_error, 33);
                dead = true;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float s[128];
#pragma unroll
            for (int c = 0; c < 4; c++) ts_ld32(tS + 32 * c, s + 32 * c);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            const int visible = last - j * kTRows;  // columns 0 .. visible of this tile
            if (visible < kTRows - 1) {
#pragma unroll
                for (int c = 0; c < 128; c++) s[c] = c <= visible ? s[c] : -INFINITY;
            }
            float t0 = s[0], t1 = s[1], t2 = s[2], t3 = s[3];
#pragma unroll
            for (int c = 4; c < 128; c += 4) {
                t0 = fmaxf(t0, s[c]); t1 = fmaxf(t1, s[c + 1]); t2 = fmaxf(t2, s[c + 2]); t3 = fmaxf(t3, s[c + 3]);
            }
            const float tile_max = fmaxf(fmaxf(t0, t1), fmaxf(t2, t3));
            // a vector's first tile always holds a visible row (row 0), later ones may hold none (tile_max = -inf); a visible
            // score may be -inf too (a product beyond the fp32 range), whose probability is 0
            if (j == 0) {
                mx = tile_max;
            } else if (__any_sync(0xffffffffu, (tile_max - mx) * kLog2e > 8.f)) {
                const float next = fmaxf(mx, tile_max);
                const float corr = next == -INFINITY ? 1.f : exp2f((mx - next) * kLog2e);
                mx = next;
                sum *= corr;
#pragma unroll 1
                for (int c = 0; c < 4; c++) {
                    float o[32];
                    ts_ld32(tO + 32 * c, o);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 32; i++) o[i] *= corr;
                    ts_st32(tO + 32 * c, reinterpret_cast<uint32_t*>(o));
                }
            }
            const float base = mx == -INFINITY ? 0.f : mx * kLog2e;
            float a0 = 0.f, a1 = 0.f;
#pragma unroll
            for (int c = 0; c < 4; c++) {
                uint32_t r[32];  // high parts, low parts of 32 probabilities
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    float e0, e1;
                    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(fmaf(s[32 * c + 2 * i], kLog2e, -base)));
                    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(fmaf(s[32 * c + 2 * i + 1], kLog2e, -base)));
                    a0 += e0;
                    a1 += e1;
                    ts_split(e0, e1, r[i], r[16 + i]);
                }
                ts_st32(tS + 32 * c, r);
            }
            sum += a0 + a1;
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) ts_arrive(&p_ready[w]);
        }
        if (!dead && !ts_wait(&o_ready[w], 0, p.spins)) {
            atomicExch(&g_prefill_wait_error, 34);
            dead = true;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (!dead) {
            const float inv = sum > 0.f ? 1.f / sum : 0.f;
            // through this tile's (finished) q rows, so that whole rows are written: chunk c of row r lies at c ^ (r % 32)
            const uint32_t sO = sQ + w * kTQ + (warp & 3) * 32 * 512;
#pragma unroll 1
            for (int c = 0; c < 4; c++) {
                float o[32];
                ts_ld32(tO + 32 * c, o);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int i = 0; i < 8; i++)
                    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(sO + lane * 512 + (((8 * c + i) ^ lane) << 4)), "f"(o[4 * i] * inv),
                                 "f"(o[4 * i + 1] * inv), "f"(o[4 * i + 2] * inv), "f"(o[4 * i + 3] * inv)
                                 : "memory");
            }
            __syncwarp();
            const int v0 = vec0 + w * 128 + (warp & 3) * 32;
#pragma unroll 4
            for (int r = 0; r < 32 && v0 + r < n_vec; r++) {
                float4 x;
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"(sO + r * 512 + ((lane ^ r) << 4)));
                reinterpret_cast<float4*>(p.out + vector_at(v0 + r))[lane] = x;
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

using EncodeTiledFp = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
bool encode_cache_map(CUtensorMap* out, const uint16_t* cache, int heads, int max_seq, int rows) {
    static EncodeTiledFp fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
        return reinterpret_cast<EncodeTiledFp>(f);
    }();
    if (!fn) return false;
    const cuuint64_t dims[3] = {cuuint64_t(kTD), cuuint64_t(rows), cuuint64_t(heads)};
    const cuuint64_t strides[2] = {cuuint64_t(kTD) * 2, cuuint64_t(max_seq) * kTD * 2};
    const cuuint32_t box[3] = {64, kTRows, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<uint16_t*>(cache), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

static int g_prefill_spins = kTSpin, g_prefill_drop = -1;  // tuning keys "prefill_wait_spins", "prefill_drop_tile" (tests of the bounded waits)
void flash_prefill_tc_set_tuning(const char* key, int value) {
    if (!strcmp(key, "prefill_wait_spins")) g_prefill_spins = value < 1 ? kTSpin : value;
    if (!strcmp(key, "prefill_drop_tile")) g_prefill_drop = value;
}

// the code of the last wait that ran out, 0 if none did since the last call; *read = false if the word cannot be read
int flash_prefill_tc_status(bool* read) {
    int v = 0;
    const int zero = 0;
    *read = cudaMemcpyFromSymbol(&v, g_prefill_wait_error, sizeof(int)) == cudaSuccess;
    if (*read && v != 0) cudaMemcpyToSymbol(g_prefill_wait_error, &zero, sizeof(int));  // reported once
    return v;
}

// false: the tensor maps cannot be made (the caller takes its other kernel)
bool flash_prefill_tc_launch(const float* q, const uint16_t* kcache, const uint16_t* vcache, float* out, int M, int Nq, int Nkv, int max_seq,
                             int n_slots, int pos0, int slot, cudaStream_t stream, int* rc) {
    PrefillTcCall c;
    memset(&c, 0, sizeof(c));
    if (!encode_cache_map(&c.k_map, kcache, n_slots * Nkv, max_seq, pos0 + M) || !encode_cache_map(&c.v_map, vcache, n_slots * Nkv, max_seq, pos0 + M))
        return false;
    c.q = q;
    c.out = out;
    c.M = M; c.Nq = Nq; c.Nkv = Nkv; c.pos0 = pos0;
    c.head0 = slot * Nkv;
    c.R = Nq / Nkv;
    c.spins = g_prefill_spins;
    c.drop = g_prefill_drop;
    static size_t configured[kMaxDevices] = {};
    if (!ensure_dynamic_smem(flash_prefill_tc_kernel, kTSmem, configured)) {
        set_error("flash_prefill: cannot reserve %zu bytes of shared memory", kTSmem);
        *rc = KUIPER_INTERNAL_ERROR;
        return true;
    }
    *rc = pdl_status(launch_pdl(flash_prefill_tc_kernel, dim3((M * c.R + 255) / 256, Nkv), dim3(kTThreads), kTSmem, stream, c), "flash_prefill");
    return true;
}

}  // namespace kuiper

// INT4-AWQ projection of a few token rows (decode batches, short prompts): y[M,N] (+)= x[M,K] . dequant(qweight)[K,N]
// for two to 32 rows, where the operation should be bound by reading the weights (4096 x 24576, ten matrices in turn so that
// they come from memory: 8 rows 13.8 us, 3.8 TB/s; four-row passes of the GEMV took 27.5, the 128-row tensor-core tiles 45.7).
// Same placeholder as the GEMV: kuiper/include/op/matmul.h:1-11 of the reference.
//
// One packed word costs six integer instructions whatever the number of rows.  Two words of consecutive weight rows
// are first merged half by half (PRMT), so that one AND isolates the same column of rows k and k + 1 in the two
// halves of a register; read as fp16 that is (q_k, q_k+1) * 2^-24 (or * 2^-20 for the high nibbles), exact subnormals.
// Those registers are the A fragments of mma.sync.m16n8k16 - 16 output columns by 16 weight rows - and eight token
// rows fill the B operand without any padding (the GEMV's fragments hold a pair of columns and leave half of B zero,
// which is why it stops at four rows).  The zero point comes back per 128-row group,
//   sum (q - z) x = sum q x - z * sum x,
// with sum x from one more mma whose A operand is all ones, then the fp16 group scale is applied in fp32.  The products
// are exact; the tensor core adds at most eight of its steps before the sums continue in fp32 registers.
//
// Work: units of 128 weight rows x 256 columns (16 KB, one quantisation group), numbered column tile major, dealt in
// equal contiguous runs.  A CTA is four consumer warps of 64 columns each and a producer warp that keeps a ring of
// stages full (four TMA boxes of 32 rows, the group's zero words and scales, the token rows' 128 fp16 activations,
// rows 272 bytes apart so that ldmatrix is conflict-free).  Up to eight rows may come as fp32, or as gate|up rows whose
// SwiGLU is the operand: two more warps then read them and write the fp16 stage, in turns, which saves a launch of 2 to 3 us
// before a projection of 4 to 10 us.  A run that leaves a column tile adds its sums to y with
// reductions, or, where the caller needs a fixed order, writes them to a workspace slot that a second kernel adds up
// in run order.  More than 32 rows run as passes over the same weights (grid.y), which the L2 serves; the ordered form takes at
// most 128 in one launch, so that its slots stay as many whatever the number of rows.
#include <cuda.h>
#include <cstring>

#include "common.cuh"

namespace kuiper {

bool awq_weight_map(const int32_t* qweight, int K, int N, CUtensorMap* out);  // awq_gemv_mma.cu

namespace {

constexpr int kTileCols = 256;
constexpr int kTileWords = kTileCols / 8;
constexpr int kGroupRows = 128;
constexpr int kWeightBytes = kGroupRows * kTileWords * 4;  // 16 KB
constexpr int kBoxRows = 32;                               // rows of one TMA box
constexpr int kZeroBytesR = kTileWords * 4;
constexpr int kScaleBytesR = kTileCols * 2;
constexpr int kXPitch = kGroupRows * 2 + 16;
constexpr int kConsumerWarps = 4;
constexpr int kThreadsRows = (kConsumerWarps + 1) * 32;
enum RowsOperand { kRowsF16, kRowsF32, kRowsSwiglu };
constexpr int rows_threads(int operand) { return kThreadsRows + (operand == kRowsF16 ? 0 : 64); }
constexpr int kPollsRows = 4096;         // polls of one round of a wait, about a microsecond each
constexpr int kRoundLimitRows = 1024;    // rounds of one wait

__device__ int g_rows_wait_error = 0;

struct RowsCall {
    CUtensorMap tmap;
    const __half* x;        // [M, K]
    const float* x32;       // the other operands: [M, K], or [M, 2 K] gate|up rows
    const uint32_t* qz;     // [K/128, N/8]
    const __half* scales;   // [K/128, N]
    float* y;               // [M, N]
    const float* residual;  // added by the run that holds a tile's first group (reductions only)
    float* partial;         // ordered: slot (run + tile) of [M][256] floats
    int M, K, N;
    int groups;             // K / 128
    int units;              // column tiles * groups
    int run;                // units per CTA
    int rounds;             // rounds after which a wait gives up
    int drop;               // test aid: this unit of every CTA is never fetched (-1: none)
};

__device__ __forceinline__ uint32_t rsm(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }
// (the limit of a call is looked at once a round: in every poll it cost 32 rows of 4096 x 24576 1.5 %, 31.7 us against 32.2)
__device__ __forceinline__ bool rows_wait(uint32_t bar, uint32_t parity, bool relaxed, const int& rounds) {
    int round = 0;
    for (int poll = 0;; poll++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if (relaxed) __nanosleep(32);
        if (poll == kPollsRows) {
            if (++round >= rounds) return false;
            poll = 0;
        }
    }
}
__device__ __forceinline__ void rows_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ uint32_t rows_lds(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void rows_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NT: eight-row blocks of token rows per pass
template <int NT>
constexpr int rows_aux_bytes() { return kZeroBytesR + kScaleBytesR + 8 * NT * kXPitch; }

template <int NT, int STAGES, int OCC, bool ORDERED, int OPERAND>
__global__ void __launch_bounds__(rows_threads(OPERAND), OCC) awq_rows_kernel(const __grid_constant__ RowsCall p) {
    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem = (rsm(smem_raw) + 1023u) & ~1023u;
    __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES];
    constexpr int kAux = rows_aux_bytes<NT>();
    const uint32_t aux0 = smem + STAGES * kWeightBytes;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int u0 = int(blockIdx.x) * p.run;
    const int n_units = min(p.run, p.units - u0);
    const int m0 = int(blockIdx.y) * 8 * NT;
    const int rows = min(8 * NT, p.M - m0);

    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < STAGES; i++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(rsm(&full_bar[i])), "n"(OPERAND == kRowsF16 ? 1 : 2));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(rsm(&empty_bar[i])), "n"(kConsumerWarps));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_launch_dependents();

    if (warp == kConsumerWarps) {
        // ------------------------------------------------------------ producer
        const int words_per_row = p.N >> 3;
        auto issue_weights = [&](int i, int s) {
            const int u = u0 + i, tile = u / p.groups, group = u - tile * p.groups;
            if (lane == 0 && i != p.drop) {
                const int cols = min(kTileCols, p.N - tile * kTileCols);
                const uint32_t zbytes = uint32_t(cols) >> 1, sbytes = uint32_t(cols) * 2;
                const uint32_t bar = rsm(&full_bar[s]), w = smem + s * kWeightBytes, aux = aux0 + s * kAux;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                             "r"(uint32_t(kWeightBytes) + zbytes + sbytes + (OPERAND == kRowsF16 ? uint32_t(rows) * kGroupRows * 2 : 0u))
                             : "memory");
#pragma unroll
                for (int b = 0; b < kGroupRows / kBoxRows; b++)
                    asm volatile(
                        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                        ::"r"(w + b * kBoxRows * kTileWords * 4), "l"(&p.tmap), "r"(tile * kTileWords), "r"(group * kGroupRows + b * kBoxRows),
                        "r"(bar)
                        : "memory");
                rows_bulk(aux, p.qz + size_t(group) * words_per_row + tile * kTileWords, zbytes, bar);
                rows_bulk(aux + kZeroBytesR, p.scales + size_t(group) * p.N + tile * kTileCols, sbytes, bar);
            }
            __syncwarp();
        };
        auto issue_x = [&](int i, int s) {
            if constexpr (OPERAND != kRowsF16) return;
            const int u = u0 + i, group = u % p.groups;
            if (lane < rows && i != p.drop)
                rows_bulk(aux0 + s * kAux + kZeroBytesR + kScaleBytesR + lane * kXPitch,
                          p.x + size_t(m0 + lane) * p.K + group * kGroupRows, kGroupRows * 2, rsm(&full_bar[s]));
            __syncwarp();
        };
        // the weights do not depend on the preceding kernel, the activations do
        const int ahead = min(STAGES, n_units);
        for (int i = 0; i < ahead; i++) issue_weights(i, i);
        if constexpr (OPERAND == kRowsF16) pdl_wait();
        for (int i = 0; i < ahead; i++) issue_x(i, i);
        int issued = ahead;
        for (; issued < n_units; issued++) {
            const int s = issued % STAGES;
            if (!rows_wait(rsm(&empty_bar[s]), uint32_t(issued / STAGES - 1) & 1u, true, p.rounds)) {
                if (lane == 0) atomicExch(&g_rows_wait_error, 11);
                break;
            }
            issue_weights(issued, s);
            issue_x(issued, s);
        }
        // The copies in flight have to land before the CTA gives its shared memory back, whoever's wait ran out: consumers that
        // gave up no longer wait for them.  Otherwise this costs nothing, the consumers wait for the same copies.
        for (int j = max(issued - STAGES, 0); j < issued; j++) rows_wait(rsm(&full_bar[j % STAGES]), uint32_t(j / STAGES) & 1u, true, p.rounds);
        return;
    }

    if constexpr (OPERAND != kRowsF16) {
        if (warp > kConsumerWarps) {
            // -------------------------------------------------------- fp32 rows: the two warps take alternate stages
            pdl_wait();
            for (int i = warp - kConsumerWarps - 1; i < n_units; i += 2) {
                const int s = i % STAGES, group = (u0 + i) % p.groups;
                float4 v[8 * NT];
#pragma unroll
                for (int r = 0; r < 8 * NT; r++) {
                    const int m = m0 + min(r, rows - 1);
                    if constexpr (OPERAND == kRowsSwiglu) {
                        const float* src = p.x32 + size_t(m) * 2 * p.K + group * kGroupRows + lane * 4;
                        const float4 g = __ldcg(reinterpret_cast<const float4*>(src)), u = __ldcg(reinterpret_cast<const float4*>(src + p.K));
                        v[r] = make_float4((g.x / (1.0f + expf(-g.x))) * u.x, (g.y / (1.0f + expf(-g.y))) * u.y,
                                           (g.z / (1.0f + expf(-g.z))) * u.z, (g.w / (1.0f + expf(-g.w))) * u.w);
                    } else {
                        v[r] = __ldcg(reinterpret_cast<const float4*>(p.x32 + size_t(m) * p.K + group * kGroupRows + lane * 4));
                    }
                }
                // a warp sees every other stage of the ring; the wait on the parity is safe because the consumers free the stages
                // in order and this warp has seen the stage before last filled
                if (i >= STAGES && !rows_wait(rsm(&empty_bar[s]), uint32_t(i / STAGES - 1) & 1u, true, p.rounds)) {
                    if (lane == 0) atomicExch(&g_rows_wait_error, 13);
                    return;
                }
                const uint32_t dst = aux0 + s * kAux + kZeroBytesR + kScaleBytesR + lane * 8;
#pragma unroll
                for (int r = 0; r < 8 * NT; r++) {
                    const __half2 a = __floats2half2_rn(v[r].x, v[r].y), b = __floats2half2_rn(v[r].z, v[r].w);
                    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst + r * kXPitch), "r"(*reinterpret_cast<const uint32_t*>(&a)),
                                 "r"(*reinterpret_cast<const uint32_t*>(&b))
                                 : "memory");
                }
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(rsm(&full_bar[s])) : "memory");
            }
            return;
        }
    }

    // ---------------------------------------------------------------- consumers: 64 columns each
    pdl_wait();
    const int g = lane >> 2, t = lane & 3;
    // word (row r, word column c) of the swizzled tile lies at r * 128 + (((c >> 2) ^ (r & 7)) << 4) + (c & 3) * 4; this lane
    // reads column 8 * warp + g of rows 2t, 2t + 1 (+ 8 j)
    const int wc = 8 * warp + g;
    const uint32_t off_even = uint32_t(2 * t) * 128 + uint32_t(((wc >> 2) ^ (2 * t)) << 4) + uint32_t(wc & 3) * 4;
    const uint32_t off_odd = uint32_t(2 * t + 1) * 128 + uint32_t(((wc >> 2) ^ (2 * t + 1)) << 4) + uint32_t(wc & 3) * 4;
    // ldmatrix: lane l addresses row l % 8 of the 8 x 8 block of k octet l / 8
    const uint32_t off_x = kZeroBytesR + kScaleBytesR + uint32_t(lane & 7) * kXPitch + uint32_t(lane >> 3) * 16;

    float acc[4][NT][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int r = 0; r < 4; r++) acc[i][n][r] = 0.f;

    int tile = u0 / p.groups, group = u0 - tile * p.groups;
    bool first_group = group == 0;  // the run holds the first group of the tile it is working on
    for (int i = 0; i < n_units; i++) {
        const int s = i % STAGES;
        if (!rows_wait(rsm(&full_bar[s]), uint32_t(i / STAGES) & 1u, false, p.rounds)) {
            if (lane == 0) atomicExch(&g_rows_wait_error, 12);
            return;  // the producer still waits for the copies in flight
        }
        const uint32_t w = smem + s * kWeightBytes, aux = aux0 + s * kAux;
        float d[4][NT][4], sum[NT][4];
#pragma unroll
        for (int n = 0; n < NT; n++) {
#pragma unroll
            for (int r = 0; r < 4; r++) sum[n][r] = 0.f;
#pragma unroll
            for (int c = 0; c < 4; c++)
#pragma unroll
                for (int r = 0; r < 4; r++) d[c][n][r] = 0.f;
        }
#pragma unroll
        for (int k2 = 0; k2 < 4; k2++) {  // 32 weight rows
            uint32_t b[NT][4];
#pragma unroll
            for (int n = 0; n < NT; n++)
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                             : "=r"(b[n][0]), "=r"(b[n][1]), "=r"(b[n][2]), "=r"(b[n][3])
                             : "r"(aux + off_x + n * 8 * kXPitch + k2 * 64));
#pragma unroll
            for (int h = 0; h < 2; h++) {  // 16 weight rows
                const uint32_t base = w + (k2 * 2 + h) * 2048;
                const uint32_t w0 = rows_lds(base + off_even), w1 = rows_lds(base + off_odd);
                const uint32_t w2 = rows_lds(base + off_even + 1024), w3 = rows_lds(base + off_odd + 1024);
                uint32_t pl = __byte_perm(w0, w1, 0x5410), ph = __byte_perm(w0, w1, 0x7632);
                uint32_t ql = __byte_perm(w2, w3, 0x5410), qh = __byte_perm(w2, w3, 0x7632);
                constexpr uint32_t kLo = 0x000f000fu, kHi = 0x00f000f0u;
#pragma unroll
                for (int n = 0; n < NT; n++) rows_mma(sum[n], 0x3c003c00u, 0x3c003c00u, 0x3c003c00u, 0x3c003c00u, b[n][2 * h], b[n][2 * h + 1]);
#pragma unroll
                for (int n = 0; n < NT; n++) rows_mma(d[0][n], pl & kLo, ph & kLo, ql & kLo, qh & kLo, b[n][2 * h], b[n][2 * h + 1]);
#pragma unroll
                for (int n = 0; n < NT; n++) rows_mma(d[1][n], pl & kHi, ph & kHi, ql & kHi, qh & kHi, b[n][2 * h], b[n][2 * h + 1]);
                pl >>= 8; ph >>= 8; ql >>= 8; qh >>= 8;
#pragma unroll
                for (int n = 0; n < NT; n++) rows_mma(d[2][n], pl & kLo, ph & kLo, ql & kLo, qh & kLo, b[n][2 * h], b[n][2 * h + 1]);
#pragma unroll
                for (int n = 0; n < NT; n++) rows_mma(d[3][n], pl & kHi, ph & kHi, ql & kHi, qh & kHi, b[n][2 * h], b[n][2 * h + 1]);
            }
        }
        // ---- group end: acc += s * (sum q x - z * sum x); rows g / g + 8 of block c are columns 2c and 2c + 1
        const uint32_t zw = rows_lds(aux + wc * 4);
        uint32_t sw[4];
        asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(sw[0]), "=r"(sw[1]), "=r"(sw[2]), "=r"(sw[3]) : "r"(aux + kZeroBytesR + wc * 16));
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(rsm(&empty_bar[s])) : "memory");
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const float unit = (c & 1) ? 0x1p-20f : 0x1p-24f, inv = (c & 1) ? 0x1p20f : 0x1p24f;
            const float z0 = -float((zw >> (4 * c)) & 15u) * unit, z1 = -float((zw >> (16 + 4 * c)) & 15u) * unit;
            const float2 sf = __half22float2(*reinterpret_cast<__half2*>(&sw[c]));
            const float s0 = sf.x * inv, s1 = sf.y * inv;
#pragma unroll
            for (int n = 0; n < NT; n++) {
                acc[c][n][0] = fmaf(fmaf(z0, sum[n][0], d[c][n][0]), s0, acc[c][n][0]);
                acc[c][n][1] = fmaf(fmaf(z0, sum[n][1], d[c][n][1]), s0, acc[c][n][1]);
                acc[c][n][2] = fmaf(fmaf(z1, sum[n][0], d[c][n][2]), s1, acc[c][n][2]);
                acc[c][n][3] = fmaf(fmaf(z1, sum[n][1], d[c][n][3]), s1, acc[c][n][3]);
            }
        }
        const bool tile_ends = ++group == p.groups;
        if (!tile_ends && i + 1 < n_units) continue;
        // ---- the run leaves this column tile: lane (g, t) holds the eight columns of word column wc for tokens 2t, 2t + 1
        const int col = tile * kTileCols + wc * 8;
        if (col < p.N) {
#pragma unroll
            for (int n = 0; n < NT; n++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int m = n * 8 + 2 * t + e;
                    if (m < rows) {
                        float4 v[2] = {make_float4(acc[0][n][e], acc[0][n][2 + e], acc[1][n][e], acc[1][n][2 + e]),
                                       make_float4(acc[2][n][e], acc[2][n][2 + e], acc[3][n][e], acc[3][n][2 + e])};
                        if constexpr (ORDERED) {
                            float4* dst = reinterpret_cast<float4*>(p.partial + (size_t(int(blockIdx.x) + tile) * p.M + m0 + m) * kTileCols + wc * 8);
                            dst[0] = v[0];
                            dst[1] = v[1];
                        } else {
                            const size_t at = size_t(m0 + m) * p.N + col;
#pragma unroll
                            for (int q = 0; q < 2; q++) {
                                if (p.residual && first_group) {
                                    const float4 r = __ldcg(reinterpret_cast<const float4*>(p.residual + at) + q);
                                    v[q].x += r.x; v[q].y += r.y; v[q].z += r.z; v[q].w += r.w;
                                }
                                asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p.y + at + 4 * q), "f"(v[q].x), "f"(v[q].y),
                                             "f"(v[q].z), "f"(v[q].w)
                                             : "memory");
                            }
                        }
                    }
                }
        }
#pragma unroll
        for (int c = 0; c < 4; c++)
#pragma unroll
            for (int n = 0; n < NT; n++)
#pragma unroll
                for (int r = 0; r < 4; r++) acc[c][n][r] = 0.f;
        if (tile_ends) {
            tile++;
            group = 0;
            first_group = true;
        }
    }
}

// y[m, 4f .. 4f+3] = residual + the slots of the runs that worked on the column's tile, in run order
__global__ void __launch_bounds__(64) awq_rows_combine_kernel(const float* __restrict__ partial, const float* residual, float* y, int M, int N,
                                                              int groups, int run) {
    pdl_launch_dependents();
    pdl_wait();
    const int f = int(blockIdx.x) * 64 + int(threadIdx.x), m = int(blockIdx.y), col = 4 * f;
    if (col >= N) return;
    const int tile = col / kTileCols;
    const int first = tile * groups / run, last = ((tile + 1) * groups - 1) / run;
    const float* base = partial + (size_t(first + tile) * M + m) * kTileCols + (col - tile * kTileCols);
    const size_t step = size_t(M) * kTileCols;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int c = first; c <= last; c++, base += step) {
        const float4 v = __ldcg(reinterpret_cast<const float4*>(base));
        sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
    }
    const size_t at = size_t(m) * N + col;
    if (residual) {
        const float4 r = __ldcg(reinterpret_cast<const float4*>(residual + at));
        sum.x += r.x; sum.y += r.y; sum.z += r.z; sum.w += r.w;
    }
    *reinterpret_cast<float4*>(y + at) = sum;
}

struct RowsPlan {
    int nt, passes, occ, tiles, groups, units, run, ctas;
};
int g_rows_min_run = 1;  // tuning key "rows_min_run"
int g_rows_rounds = kRoundLimitRows, g_rows_drop = -1;  // tuning keys "rows_wait_spins" (polls), "rows_drop_unit": tests of the bounded waits
// four passes (51 rows of 3456 x 96, whose launches are what counts: 11.2 us; in blocks of 32 rows 18.8)
constexpr int kOrderedRows = 128;

RowsPlan plan_rows(int M, int K, int N, bool ordered) {
    RowsPlan r;
    r.nt = M <= 8 ? 1 : (M <= 16 ? 2 : 4);
    r.passes = (M + 8 * r.nt - 1) / (8 * r.nt);
    r.tiles = (N + kTileCols - 1) / kTileCols;
    r.groups = K / kGroupRows;
    r.units = r.tiles * r.groups;
    // (one matrix over and over, which stays in the L2)
    // Three CTAs per SM stream a large matrix faster (4096 x 24576, 8 rows: 14.8 us against 15.6 with two, 16 rows 17.2 / 19.2).
    // A small one is faster with two, whose runs fill a deeper ring (2560 x 6144, 8 rows: 4.1 us against 4.8, 16 rows 5.7 / 6.2;
    // 9728 x 2560 5.8 / 6.2, 7.9 / 8.4) - but up to eight rows three leave the next launch of a decode step more room (Qwen3-8B,
    // five sequences: 50.2 ms for 24 steps against 53.1), so there only the ordered form does that.  32 rows need the registers
    // of two.
    r.occ = r.nt == 4 || (r.units * r.passes <= 800 && (ordered || r.nt == 2)) ? 2 : 3;
    const int slots = device_sm_count() * r.occ;
    r.run = int(((long long)r.units * r.passes + slots - 1) / slots);
    if (r.run < g_rows_min_run) r.run = g_rows_min_run;
    r.ctas = (r.units + r.run - 1) / r.run;
    return r;
}

template <int NT, int STAGES, int OCC, bool ORDERED, int OPERAND>
int launch_rows(const RowsCall& call, const RowsPlan& plan, cudaStream_t stream) {
    auto kern = awq_rows_kernel<NT, STAGES, OCC, ORDERED, OPERAND>;
    const size_t smem = 1024 + size_t(STAGES) * (kWeightBytes + rows_aux_bytes<NT>());
    static size_t configured[kMaxDevices] = {};
    if (!ensure_dynamic_smem(kern, smem, configured)) {
        set_error("awq_gemm: cannot reserve %zu bytes of shared memory", smem);
        return KUIPER_INTERNAL_ERROR;
    }
    return pdl_status(launch_pdl(kern, dim3(plan.ctas, plan.passes), dim3(rows_threads(OPERAND)), smem, stream, call), "awq_gemm rows");
}

template <bool ORDERED>
int launch_rows_nt(const RowsCall& call, const RowsPlan& plan, int operand, cudaStream_t stream) {
    if (operand == kRowsSwiglu) return launch_rows<1, 3, 3, false, kRowsSwiglu>(call, plan, stream);
    if constexpr (ORDERED) {
        if (operand == kRowsF32 && plan.occ == 2) return launch_rows<1, 5, 2, true, kRowsF32>(call, plan, stream);
    }
    if (operand == kRowsF32) return launch_rows<1, 3, 3, ORDERED, kRowsF32>(call, plan, stream);
    if constexpr (ORDERED) {
        if (plan.nt == 1 && plan.occ == 2) return launch_rows<1, 5, 2, true, kRowsF16>(call, plan, stream);
    }
    if (plan.nt == 2 && plan.occ == 2) return launch_rows<2, 4, 2, ORDERED, kRowsF16>(call, plan, stream);
    if (plan.nt == 1) return launch_rows<1, 3, 3, ORDERED, kRowsF16>(call, plan, stream);
    if (plan.nt == 2) return launch_rows<2, 3, 3, ORDERED, kRowsF16>(call, plan, stream);
    return launch_rows<4, 3, 2, ORDERED, kRowsF16>(call, plan, stream);
}

bool fill_rows(RowsCall& call, const RowsPlan& plan, const __half* x16, const int32_t* qweight, const int32_t* qzeros, const uint16_t* scales,
               float* y, int M, int K, int N) {
    memset(&call, 0, sizeof(call));
    if (!awq_weight_map(qweight, K, N, &call.tmap)) return false;
    call.x = x16;
    call.qz = reinterpret_cast<const uint32_t*>(qzeros);
    call.scales = reinterpret_cast<const __half*>(scales);
    call.y = y;
    call.M = M; call.K = K; call.N = N;
    call.groups = plan.groups;
    call.units = plan.units;
    call.run = plan.run;
    call.rounds = g_rows_rounds;
    call.drop = g_rows_drop;
    return true;
}

}  // namespace

void awq_rows_set_tuning(const char* key, int value) {
    if (!strcmp(key, "rows_min_run")) g_rows_min_run = value < 1 ? 1 : value;
    if (!strcmp(key, "rows_wait_spins")) g_rows_rounds = value < 1 ? kRoundLimitRows : (value - 1) / kPollsRows + 1;
    if (!strcmp(key, "rows_drop_unit")) g_rows_drop = value;
}

int awq_rows_status() {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_rows_wait_error, sizeof(int)) != cudaSuccess) return -1;
    return v;
}

// y += x16 . W (+ residual); y holds the addend.  Needs N % 32 == 0 and 16-byte aligned tensors.
int awq_rows_launch(const __half* x16, const int32_t* qweight, const int32_t* qzeros, const uint16_t* scales, float* y, const float* residual,
                    int M, int K, int N, cudaStream_t stream) {
    const RowsPlan plan = plan_rows(M, K, N, false);
    RowsCall call;
    if (!fill_rows(call, plan, x16, qweight, qzeros, scales, y, M, K, N)) {
        set_error("awq_gemm: tensor map encoding failed");
        return KUIPER_INTERNAL_ERROR;
    }
    call.residual = residual;
    return launch_rows_nt<false>(call, plan, kRowsF16, stream);
}

// most rows of awq_rows_f32_launch
int awq_rows_f32_max() { return 8; }

// y += op(x) . W for fp32 rows; op: fp16 rounding, or (swiglu) silu(gate) * up of [M, 2 K] rows rounded to fp16
int awq_rows_f32_launch(const float* x, bool swiglu, const int32_t* qweight, const int32_t* qzeros, const uint16_t* scales, float* y, int M, int K,
                        int N, cudaStream_t stream) {
    const RowsPlan plan = plan_rows(M, K, N, false);
    RowsCall call;
    if (!fill_rows(call, plan, nullptr, qweight, qzeros, scales, y, M, K, N)) {
        set_error("awq_gemv: tensor map encoding failed");
        return KUIPER_INTERNAL_ERROR;
    }
    call.x32 = x;
    return launch_rows_nt<false>(call, plan, swiglu ? kRowsSwiglu : kRowsF32, stream);
}

// most rows of awq_rows_ordered_launch
int awq_rows_ordered_max() { return kOrderedRows; }

// floats of the slots that ordered calls of up to M rows write: the most that any of them needs (two CTAs per SM have fewer
// slots than three, so 17 rows may need less than 16)
size_t awq_rows_partial_floats(int M, int K, int N) {
    size_t most = 0;
    // the largest call of each plan: 8 or 16 rows, or a number of 32-row passes
    for (int m = M < kOrderedRows ? M : kOrderedRows; m > 0; m = m > 32 ? (m - 1) / 32 * 32 : (m > 16 ? 16 : (m > 8 ? 8 : 0))) {
        const RowsPlan plan = plan_rows(m, K, N, true);
        const size_t floats = size_t(plan.ctas + plan.tiles) * m * kTileCols;
        if (floats > most) most = floats;
    }
    return most;
}

// y = x . W (+ residual) with a fixed summation order for up to awq_rows_ordered_max rows, x as fp16 (x16) or, up to
// awq_rows_f32_max rows, fp32; partial: awq_rows_partial_floats floats
int awq_rows_ordered_launch(const __half* x16, const float* x32, const int32_t* qweight, const int32_t* qzeros, const uint16_t* scales, float* y,
                            const float* residual, float* partial, int M, int K, int N, cudaStream_t stream) {
    const RowsPlan plan = plan_rows(M, K, N, true);
    RowsCall call;
    if (!fill_rows(call, plan, x16, qweight, qzeros, scales, y, M, K, N)) {
        set_error("awq_gemv: tensor map encoding failed");
        return KUIPER_INTERNAL_ERROR;
    }
    call.partial = partial;
    call.x32 = x32;
    const int rc = launch_rows_nt<true>(call, plan, x32 ? kRowsF32 : kRowsF16, stream);
    if (rc != KUIPER_OK) return rc;
    return pdl_status(launch_pdl(awq_rows_combine_kernel, dim3((N / 4 + 63) / 64, M), dim3(64), 0, stream, static_cast<const float*>(partial), residual, y,
                                 M, N, plan.groups, plan.run),
                      "awq_gemv combine");
}

}  // namespace kuiper

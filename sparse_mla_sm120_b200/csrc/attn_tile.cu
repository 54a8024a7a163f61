// Sparse-MLA attention of up to 64 query heads over packed 656-byte rows (sm_100a): split-KV decode and prefill, one CTA per
// partition (a run of 64-token blocks of consecutive requests, see sched.cu; without a scheduler every parts-th request).
//
// Why not two CTAs as in attn_pair.cu and attn_duo.cu: they spend both on a partition whatever the number of heads and split the work
// over half as many partitions.  48 requests of top-k 2048 at 16 heads: 45.1 us in attn_pair_kernel, 28.0 us here; 1237 ragged prompt
// tokens of top-k 1024 at 64 heads: 395 us there, 163 us here.  At 128 heads two of these CTAs would gather every row twice: 2400 us for
// 4096 tokens of top-k 2048, against 1815 us in attn_duo_kernel.
//
// What bounds it: no unit is near its limit (ncu, 592 tokens of 2048 entries at 64 heads, rows in HBM: issue slots 43 %, ALU pipe 32 %,
// tensor pipe 22 %, 3.1 TB/s); a tile waits for its own way through the SM.  Its parts (clock64 at 64 heads, 1.9 GHz, before the copies
// were issued from indices in shared memory and the MMAs from loops, which took 48 requests from 32.8 to 30.7 us and the ragged
// prompt from 175 to 165): a tile of 128 tokens takes 4300 cycles, half of the way of a tile from the load of its rows (2000 cycles: the gather delivers 35 bytes per cycle and SM) over its scores (2100, with the hand-overs) and its
// weights (2700) to P.V (1300), because two tiles are all that shared memory holds.  A request costs another 15000 cycles for its
// q and its epilogue, which the softmax warps do in between.  Tried without gain: sixteen softmax warps (2485 us where
// eight take 2400), q and epilogue on four warps of their own (169 us for the
// ragged prompt, but 36.8 us for the 48 requests: every role's code grows, and code beyond the instruction caches slows all of
// them; fully unrolled gathers and MMAs 188 us), weights before the group's barrier (2483), a tighter rescale threshold (3350, more rescales).
//
// The gathered rows are never touched by a thread.  TMA gather4 loads bring the 512 e4m3 values of a row, as four
// pieces of 128 dims, and its 64 RoPE values straight into the 128B-swizzled tiles that the MMAs read; a row without an
// entry is named by an index outside the tensor and arrives as zeros.  Both contractions run transposed, with the tile of
// rows as the A operand of both (M = 128 whatever the number of heads, and V needs no second copy):
//   * S^T [128 tokens x 64 heads] = K . Q^T, K-major.  The four fp32 scales of a row (powers of two, one per 128 dims) and
//     the scale of a head's quantised q are applied by the tensor core: kind::mxf8f6f4 takes one power of two per row and 32
//     values, and the scale bytes of a row's four blocks are the four bytes of one scale word.  RoPE follows as bf16 MMAs
//     into the same accumulator, so the accumulator holds q . k itself.
//   * O^T [4 x 128 dims x 64 heads] += V^T . P_b, the same tile read MN-major.  V's scale is a factor of the token inside a
//     block of 128 dims, so it goes into the weights: block b uses P_b = P' * 2^(e_b - e_g + k_b), rounded to e4m3, with
//     e_g the largest exponent of the token's group of eight (the group of the pair kernel, so that P' is its P') and k_b,
//     the same for all tokens of a request, as large as it can be without lifting any P_b over P'.  A block whose scales
//     are small throughout so has weights as precise as the largest block's: without k_b, scales 2^-9 below the row's
//     largest leave weights in e4m3's subnormals (error of that block 12 % at logits of +-6 instead of 0.6 %).  k_b only
//     ever falls; the block's part of the accumulator is then multiplied by the power of two (exactly), and the epilogue
//     takes 2^k_b out again.  Price: 172 -> 174.6 us for 1237 ragged prompt tokens, 2 % and less elsewhere.
// Numerics (the FP8 class of the reference's V32 kernels, which quantise Q and P to e4m3:
// csrc/kernel/common/fp8_quant.cuh:44-103, csrc/kernel/decode/decode_v2_kernel.cuh:414-493): q no-PE e4m3 with one power of
// two per head, q RoPE bf16 as given, K and V bytes as stored, P' = 2^(z - m) in e4m3 (times 2^T_P_SHIFT) with
// z = logit * log2(e) + e_g and m its lazily updated running maximum per head; the denominator sums P' / 2^e_g in fp32.
// Entries without a row (index < 0, position >= topk_length) have weight exactly 0.
//
// Warp roles (640 threads):
//   warps 0-7    softmax, epilogue, Q: warp w holds tokens [32 (w % 4), +32) and heads [32 (w / 4), +32) of a tile, a thread
//                one token; the four warps of a head half meet once per tile at a barrier that also ORs "a weight has outgrown
//                the running maximum".  Warps 4-7 only quantise Q when there are 32 heads or fewer.
//   warps 8-11   producers: warp 8 + i gathers rows [32 i, +32) of every tile; a quarter of a stage is refilled as soon as
//                P.V has read it.
//   warps 12-15  scales: the rows' scale words into tensor memory (each warp the 32 lanes it can reach) and shared memory.
//   warp 16      issues the score MMAs, warp 17 the P.V MMAs (one elected lane each).
// Every wait is bounded; a wait that gives up records a code in status[] and the CTA drains and exits.
#include "attn_common.cuh"
#include "rows_map.cuh"
#include "sm100_ptx.cuh"

namespace smla {

namespace {

using namespace ptx;
using namespace attn;

constexpr int T_HEADS = 64;                    // heads per CTA
constexpr int T_TILE = TILE_N;
constexpr int T_SM_WARPS = 8, T_PROD = 8, T_SCALE = 12, T_QK = 16, T_PV = 17;
constexpr int T_THREADS = 20 * 32;
constexpr int T_REGS_LAUNCH = 96, T_REGS_SOFTMAX = 152, T_REGS_REST = 56;
static_assert(T_SM_WARPS * 32 * T_REGS_SOFTMAX + (T_THREADS - T_SM_WARPS * 32) * T_REGS_REST <= T_THREADS * T_REGS_LAUNCH,
              "register budgets exceed what the CTA owns");
constexpr int T_P_SHIFT = 5;                   // P' is stored as e4m3(P' * 2^T_P_SHIFT)
constexpr float T_NO_MAX = 1e30f;              // minus the running maximum of a head that has seen no entry (finite: -inf minus it is -inf)
constexpr float T_TAU = 3.0f;                  // lazy-rescale threshold (log2 units); P' <= 2^T_TAU
constexpr int NSTAGE = 2;

constexpr uint32_t K_CHUNK = T_TILE * 128;                 // 128 dims (or the RoPE) of all rows
constexpr uint32_t Q_CHUNK = T_HEADS * 128;
constexpr uint32_t K_STAGE = 4 * K_CHUNK;
constexpr uint32_t K_OFF = 0;
constexpr uint32_t R_OFF = K_OFF + NSTAGE * K_STAGE;       // RoPE of the rows: one stage, free again when the scores are done
constexpr uint32_t Q_OFF = R_OFF + K_CHUNK;                // q e4m3, four chunks of [64 heads x 128 dims]
constexpr uint32_t QR_OFF = Q_OFF + 4 * Q_CHUNK;           // q RoPE bf16
constexpr uint32_t P_OFF = QR_OFF + Q_CHUNK;               // P_b: [128 tokens x 64 heads] e4m3, 64B swizzle
constexpr uint32_t P_BYTES = T_TILE * T_HEADS;
constexpr int SW_RING = 4;
constexpr uint32_t SW_OFF = P_OFF + 4 * P_BYTES;           // TokenScale of a tile's tokens, [SW_RING][128]
constexpr uint32_t NM_OFF = SW_OFF + SW_RING * T_TILE * 8; // -m of the 64 heads
constexpr uint32_t QW_OFF = NM_OFF + T_HEADS * 4;          // the heads' scale words
constexpr uint32_t XX_OFF = QW_OFF + T_HEADS * 4;          // exchange between the four warps of a head half: [2][4][64] fp32
constexpr uint32_t KX_OFF = XX_OFF + 2 * 4 * T_HEADS * 4;  // the same for the blocks' shifts: [2 halves][4]
constexpr uint32_t IDX_OFF = KX_OFF + 2 * 4 * 4;           // the rows that a producer is about to ask for: [4][32]
constexpr uint32_t WORD_OFF = IDX_OFF + 4 * 32 * 4;        // the rows' scale words on their way to tensor memory: [2][128]
constexpr uint32_t B_OFF = WORD_OFF + 2 * T_TILE * 4;
constexpr int B_KFULL = 0, B_RFULL = B_KFULL + NSTAGE, B_KFREE = B_RFULL + 1, B_SREADY = B_KFREE + 4 * NSTAGE, B_SFREE = B_SREADY + 2,
              B_SCALES = B_SFREE + 2, B_PREADY = B_SCALES + SW_RING, B_PVDONE = B_PREADY + 1, B_QREADY = B_PVDONE + 1, B_N = B_QREADY + 1;
constexpr uint32_t MISC_OFF = B_OFF + B_N * 8;
constexpr uint32_t T_SMEM = MISC_OFF + 16 + 1024;
static_assert(T_SMEM <= 227 * 1024, "shared memory budget");
static_assert(IDX_OFF % 16 == 0 && R_OFF % 1024 == 0 && Q_OFF % 1024 == 0 && P_OFF % 1024 == 0 && B_OFF % 8 == 0, "alignment");

// tensor memory: dims block b of O^T at 64 b, score buffers, scale words of the rows (4 columns per tile) and of the heads
constexpr uint32_t TM_O = 0, TM_S = 256, TM_SFA = 384, TM_SFB = 400;
// Instruction descriptors.  kind::mxf8f6f4: scale type UE8M0 (bit 23), which byte of the scale word A uses (bits 29-30); the
// head's word has the same byte four times.
__host__ __device__ constexpr uint32_t idesc_mx(uint32_t a_byte) {
    return (FMT_E4M3 << 7) | (FMT_E4M3 << 10) | ((T_HEADS >> 3) << 17) | (1u << 23) | ((T_TILE >> 7) << 27) | (a_byte << 29);
}
constexpr uint32_t IDESC_ROPE = instr_desc(FMT_BF16, FMT_BF16, false, false, T_TILE, T_HEADS);
constexpr uint32_t IDESC_PV = instr_desc(FMT_E4M3, FMT_E4M3, true, true, 128, T_HEADS);
constexpr uint32_t HI_128 = desc_hi(1024, (uint32_t)SWIZZLE_128B), HI_P = desc_hi(512, (uint32_t)SWIZZLE_64B);

enum { WT_KFULL = 51, WT_RFULL = 52, WT_KFREE = 53, WT_SREADY = 54, WT_SFREE = 55, WT_SCALES = 56, WT_PREADY = 57, WT_PVDONE = 58, WT_QREADY = 59 };

__device__ __forceinline__ uint32_t swz128(uint32_t row, uint32_t piece) { return row * 128u + ((piece ^ (row & 7u)) << 4); }
__device__ __forceinline__ uint32_t swz64(uint32_t row, uint32_t piece) { return row * 64u + ((piece ^ ((row >> 1) & 3u)) << 4); }

__device__ __forceinline__ float lanes_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// What the softmax needs of a token's scales: by how many powers of two each of its four blocks lies below e_g, the largest
// exponent of the group of eight tokens (a byte per block, at most NO_SHIFT), and e_g itself (biased; 0: no entry).
struct TokenScale { uint32_t below, e_g; };
constexpr uint32_t NO_SHIFT = 0x7fu;

template <bool MAXL>
__global__ void __launch_bounds__(T_THREADS, 1) attn_tile_kernel(const AttnParams p, const __grid_constant__ CUtensorMap kv_map) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* sm = smem_raw + (base - raw);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + MISC_OFF + 4);
    const uint32_t abort_addr = base + MISC_OFF + 4;
    auto bar = [&](int i) -> uint32_t { return base + B_OFF + 8u * i; };
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int part = blockIdx.x, my_heads = p.num_heads;   // at most T_HEADS
    const int act = my_heads > 32 ? 8 : 4;                 // softmax warps with live heads

    if (tid == 0) {
        for (int s = 0; s < NSTAGE; ++s) {
            mbar_init(bar(B_KFULL + s), 4);                // + the bytes of the four producers
            for (int i = 0; i < 4; ++i) mbar_init(bar(B_KFREE + 4 * s + i), 1);
        }
        mbar_init(bar(B_RFULL), 4);
        for (int b = 0; b < 2; ++b) { mbar_init(bar(B_SREADY + b), 1); mbar_init(bar(B_SFREE + b), act); }
        for (int i = 0; i < SW_RING; ++i) mbar_init(bar(B_SCALES + i), 4);
        mbar_init(bar(B_PREADY), act);
        mbar_init(bar(B_PVDONE), 1);
        mbar_init(bar(B_QREADY), T_SM_WARPS);
        *abort_flag = 0;
        mbar_init_fence();
    }
    if (act == 4)                                          // the weights of heads that do not exist stay zero
        for (int i = tid; i < (int)(4 * P_BYTES / 16); i += T_THREADS) reinterpret_cast<uint4*>(sm + P_OFF)[i] = make_uint4(0, 0, 0, 0);
    if (warp == T_QK) { tmem_alloc(base + MISC_OFF, 512); tmem_relinquish(); }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(sm + MISC_OFF);
    grid_dep_wait();
    grid_dep_launch();
    SchedMeta meta;
    int first, step, last;
    if (p.sched != nullptr || p.uniform_k > 1) {
        meta = load_meta(p, part);
        first = meta.begin_req; step = 1; last = min(meta.end_req, p.num_tokens - 1);
    } else {                                               // whole requests; neighbours differ little in length, so every CTA takes each parts-th
        meta.begin_block = 0; meta.end_block = 0x7fffffff;
        meta.begin_split = 0; meta.first_split = meta.last_split = 0; meta.pad = 0;
        first = part; step = (int)gridDim.x; last = p.num_tokens - 1;
        meta.begin_req = 0; meta.end_req = last;
    }
    if (warp < T_SM_WARPS) setmaxnreg_inc<T_REGS_SOFTMAX>();
    else setmaxnreg_dec<T_REGS_REST>();

    if (warp < T_SM_WARPS) {
        // =================================================================== softmax + epilogue + Q
        const int quarter = warp & 3, half = warp >> 2;
        const int token = quarter * 32 + lane;             // of the tile; in O^T: output dim inside a block of 128
        const int hl = half * 32 + lane;                   // the head whose state this lane keeps (the same in four warps)
        const bool live = hl < my_heads, active = half * 32 < my_heads;
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
        float* nm = reinterpret_cast<float*>(sm + NM_OFF);
        float* xx = reinterpret_cast<float*>(sm + XX_OFF);
        uint32_t* kx = reinterpret_cast<uint32_t*>(sm + KX_OFF);
        uint32_t* qw = reinterpret_cast<uint32_t*>(sm + QW_OFF);
        // logits in log2 units are scores times a positive number: the sign of the softmax scale goes into q
        const float c = fabsf(p.sm_scale) * LOG2E;
        const uint32_t scale_sign = __float_as_uint(p.sm_scale) & 0x80000000u;
        Walk tiles(p, first, step, last);
        uint32_t it = 0;
        bool dead = false;
        bool prev = false, prev_no_split = false;          // a request's epilogue runs after the next request's Q phase
        int prev_req = 0, prev_split = 0;
        float prev_m = 0.f, prev_l = 0.f, prev_x = 0.f;
        uint32_t prev_shift = 0u;
        while (true) {
            const bool have = tiles.next_request(p, meta);
            // Every score of the request before has been read, by all warps, and so has its state: q, its scales and the maxima may
            // be overwritten.  The eight warps leave the loop here together when one of them has given up.
            if (named_bar_or(3, T_SM_WARPS * 32, dead || *abort_flag != 0)) break;
            if (have) {
                // ---- Q: warp w quantises heads [8 w, +8), a lane 16 of the 512 no-PE dims of each
                const __nv_bfloat16* q0 = p.q + ((size_t)tiles.req * my_heads) * D_QK;
#pragma unroll 1
                for (int u = 0; u < 8; u += 4) {
                    uint4 v[8];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int h = 8 * warp + u + k;
                        v[2 * k] = v[2 * k + 1] = make_uint4(0, 0, 0, 0);
                        if (h < my_heads) {
                            v[2 * k] = ld_in(reinterpret_cast<const uint4*>(q0 + (size_t)h * D_QK + lane * 16));
                            v[2 * k + 1] = ld_in(reinterpret_cast<const uint4*>(q0 + (size_t)h * D_QK + lane * 16 + 8));
                        }
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int h = 8 * warp + u + k;
                        const uint32_t x[8] = {v[2 * k].x, v[2 * k].y, v[2 * k].z, v[2 * k].w, v[2 * k + 1].x, v[2 * k + 1].y, v[2 * k + 1].z, v[2 * k + 1].w};
                        uint32_t am = 0u;                  // magnitudes of bf16 numbers order as integers do
#pragma unroll
                        for (int i = 0; i < 8; ++i) am = __vmaxu2(am, x[i] & 0x7fff7fffu);
                        am = __reduce_max_sync(0xffffffffu, max(am & 0xffffu, am >> 16));
                        const float sq = pow2_ceil(fmaxf(__uint_as_float(am << 16), 1e-4f) * (1.f / 448.f));
                        const float is = __uint_as_float((0x7f000000u - __float_as_uint(sq)) | scale_sign);   // 1/sq, sq a power of two
                        uint32_t o[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            o[i] = pack_e4m3x4(bf16lo(x[2 * i]) * is, bf16hi(x[2 * i]) * is, bf16lo(x[2 * i + 1]) * is, bf16hi(x[2 * i + 1]) * is);
                        *reinterpret_cast<uint4*>(sm + Q_OFF + (lane >> 3) * Q_CHUNK + swz128((uint32_t)h, (uint32_t)lane & 7u)) = make_uint4(o[0], o[1], o[2], o[3]);
                        if (lane == 0) qw[h] = (__float_as_uint(sq) >> 23) * 0x01010101u;
                    }
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {              // RoPE
                    const int h = 8 * warp + 4 * u + (lane >> 3);
                    uint4 v = make_uint4(0, 0, 0, 0);
                    if (h < my_heads) v = ld_in(reinterpret_cast<const uint4*>(q0 + (size_t)h * D_QK + D_NOPE + (lane & 7) * 8));
                    const uint32_t flip = scale_sign | (scale_sign >> 16);
                    v.x ^= flip; v.y ^= flip; v.z ^= flip; v.w ^= flip;
                    *reinterpret_cast<uint4*>(sm + QR_OFF + swz128((uint32_t)h, (uint32_t)lane & 7u)) = v;
                }
                fence_proxy_async();
                if (warp < 2) nm[warp * 32 + lane] = T_NO_MAX;
                named_bar_sync(3, T_SM_WARPS * 32);
                if (half == 0) {                           // the heads' scale words, in the lanes that this warp reaches
                    const uint32_t w2[2] = {qw[lane], qw[32 + lane]};
                    tmem_st2(lane_addr + TM_SFB, w2);
                    tmem_wait_st();
                }
                tc_fence_before();                         // also orders the previous epilogue's reads of the accumulator
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(B_QREADY));
                // ask L2 for the next request's q, a whole request of tiles ahead of its use
                if (tiles.req + tiles.step <= tiles.last) {
                    const uint8_t* qn = reinterpret_cast<const uint8_t*>(p.q + ((size_t)(tiles.req + tiles.step) * my_heads) * D_QK);
                    for (int i = tid; i < (my_heads * D_QK * 2 + 127) >> 7; i += T_SM_WARPS * 32)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(qn + (size_t)i * 128));
                }
            }
            // ---- epilogue of the request before
            auto epilogue = [&]() {
                if (!dead) dead = !mbar_wait_lean(bar(B_PVDONE), (it - 1) & 1u, abort_addr, WT_PVDONE);
                tc_fence_after();
                xx[quarter * T_HEADS + hl] = prev_l;
                if (MAXL) xx[(4 + quarter) * T_HEADS + hl] = prev_x;
                if (named_bar_or(1 + half, 128, dead || *abort_flag != 0)) { dead = true; return; }
                const float l_all = (xx[hl] + xx[T_HEADS + hl]) + (xx[2 * T_HEADS + hl] + xx[3 * T_HEADS + hl]);
                float x_all = -INFINITY;
                if (MAXL) x_all = fmaxf(fmaxf(xx[256 + hl], xx[256 + T_HEADS + hl]), fmaxf(xx[256 + 2 * T_HEADS + hl], xx[256 + 3 * T_HEADS + hl]));
                float lse = (l_all > 0.f) ? (log2f(l_all) - (float)T_P_SHIFT + prev_m) : NEG_BIG;
                float denom = l_all;
                if (prev_no_split && p.attn_sink != nullptr && live) {
                    const float sink2 = p.attn_sink[hl] * LOG2E;
                    denom = l_all + ((prev_m == -T_NO_MAX) ? INFINITY : exp2f(sink2 - prev_m + (float)T_P_SHIFT));
                    if (lse != NEG_BIG) lse += log2f(1.f + exp2f(sink2 - lse));
                    else lse = sink2;
                }
                named_bar_sync(1 + half, 128);             // the sums have been read: 1 / denominator takes the place of a quarter's
                float* iv = xx + quarter * T_HEADS + half * 32;
                iv[lane] = (denom > 0.f) ? 1.f / denom : 0.f;
                __syncwarp();
                const size_t row0 = (size_t)(prev_no_split ? prev_req : prev_split) * my_heads + half * 32;
                const int n_live = min(my_heads - half * 32, 32);
                const bool odd = (lane & 1) != 0;
                const uint32_t sel0 = odd ? 0x1054u : 0x5410u, sel1 = odd ? 0x3276u : 0x7632u;
                // 1 / denominator by broadcast reads instead of a shuffle per head, one conversion per type: 6 us of 178 at 64 heads
#pragma unroll 1
                for (int b = 0; b < 4; ++b) {
                    uint32_t o[32];
                    tmem_ld32(lane_addr + TM_O + 64 * b + 32 * half, o);
                    const float unshift = __uint_as_float((127u - ((prev_shift >> (8 * b)) & 0xffu)) << 23);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; i += 4) {
                        const float4 f = *reinterpret_cast<const float4*>(iv + i);
                        o[i] = __float_as_uint(__uint_as_float(o[i]) * unshift * f.x);
                        o[i + 1] = __float_as_uint(__uint_as_float(o[i + 1]) * unshift * f.y);
                        o[i + 2] = __float_as_uint(__uint_as_float(o[i + 2]) * unshift * f.z);
                        o[i + 3] = __float_as_uint(__uint_as_float(o[i + 3]) * unshift * f.w);
                    }
                    if (!prev_no_split && p.uniform_k <= 1) {      // fp32 records: a head's 32 dims of the warp are one store of 128 bytes
                        float* dst = p.o_accum + row0 * D_V + 128 * b + token;
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (i < n_live) dst[i * D_V] = __uint_as_float(o[i]);
                        continue;
                    }
                    // 16-bit results (bf16 outputs; fp16 records of equal partitions, the library's own scratch): neighbouring lanes
                    // exchange halves, so that a lane has two dims of 16 heads (even lanes heads 0-15, odd lanes 16-31)
                    const int n = n_live - (odd ? 16 : 0);
                    uint32_t* dst = reinterpret_cast<uint32_t*>(prev_no_split ? reinterpret_cast<void*>(p.out) : reinterpret_cast<void*>(p.o_accum)) +
                                    (row0 + (odd ? 16 : 0)) * (D_V / 2) + 64 * b + (token >> 1);
                    if (prev_no_split) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const __nv_bfloat162 t = __floats2bfloat162_rn(__uint_as_float(o[2 * i]), __uint_as_float(o[2 * i + 1]));
                            o[i] = *reinterpret_cast<const uint32_t*>(&t);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const __half2 t = __floats2half2_rn(__uint_as_float(o[2 * i]), __uint_as_float(o[2 * i + 1]));
                            o[i] = *reinterpret_cast<const uint32_t*>(&t);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) {          // own: this lane's dim of two heads; got: the neighbour's
                        const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? o[i] : o[8 + i], 1), own = odd ? o[8 + i] : o[i];
                        if (2 * i < n) dst[2 * i * (D_V / 2)] = __byte_perm(own, got, sel0);
                        if (2 * i + 1 < n) dst[(2 * i + 1) * (D_V / 2)] = __byte_perm(own, got, sel1);
                    }
                }
                if (live && quarter == 0) {
                    if (prev_no_split) {
                        p.out_lse[row0 + lane] = lse;
                        if (MAXL) p.out_max_logits[row0 + lane] = (x_all == -INFINITY) ? NEG_BIG : x_all;
                    } else {
                        p.lse_accum[row0 + lane] = lse;
                    }
                }
                tc_fence_before();                         // the accumulator's reads precede the next request's first P.V
                named_bar_sync(1 + half, 128);             // xx is free again
            };
            if (prev && active) epilogue();
            prev = false;
            if (!have) break;
            if (!active) continue;                         // no heads here
            uint64_t l2[16];                               // this token's share of the denominators of the warp's 32 heads
            float xm[MAXL ? 32 : 1];
#pragma unroll
            for (int i = 0; i < 16; ++i) l2[i] = 0ull;
#pragma unroll
            for (int i = 0; i < (MAXL ? 32 : 1); ++i) xm[i] = -INFINITY;
            uint32_t shift = NO_SHIFT * 0x01010101u;       // of the four blocks; the same in all warps of the half
            for (int j = 0; j < tiles.nst; ++j, ++it) {
                const uint32_t b = it & 1u;
                uint32_t z[32];
                TokenScale ts{NO_SHIFT * 0x01010101u, 0u};
                bool grow = false;
                float off = 0.f;                           // log2 of the group's scale + T_P_SHIFT: weights carry the shift
                auto load_scores = [&]() {
                    tmem_ld32(lane_addr + TM_S + 64 * b + 32 * half, z);
                    tmem_wait_ld();
                };
                // exponents: two per packed addition and FMA
                auto exponents = [&]() {
                    const uint64_t c2 = pack_f32x2(c, c), off2 = pack_f32x2(off, off);
                    float mx = -INFINITY;
#pragma unroll
                    for (int i = 0; i < 32; i += 4) {
                        const ulonglong2 m4 = *reinterpret_cast<const ulonglong2*>(nm + half * 32 + i);
                        uint64_t a = m4.x, d = m4.y;
                        add_f32x2(a, off2);
                        add_f32x2(d, off2);
                        fma_f32x2(a, pack_f32x2(__uint_as_float(z[i]), __uint_as_float(z[i + 1])), c2);
                        fma_f32x2(d, pack_f32x2(__uint_as_float(z[i + 2]), __uint_as_float(z[i + 3])), c2);
                        float e0, e1, e2, e3;
                        unpack_f32x2(a, e0, e1);
                        unpack_f32x2(d, e2, e3);
                        mx = fmaxf(mx, fmaxf(fmaxf(e0, e1), fmaxf(e2, e3)));
                        z[i] = __float_as_uint(e0); z[i + 1] = __float_as_uint(e1); z[i + 2] = __float_as_uint(e2); z[i + 3] = __float_as_uint(e3);
                    }
                    if (!__all_sync(0xffffffffu, ts.e_g != 0u) && ts.e_g == 0u) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) z[i] = 0xff800000u;      // no entry: weight exactly 0
                    }
                    return mx;
                };
                if (!dead) dead = !mbar_wait_lean(bar(B_SCALES + (it & (SW_RING - 1))), (it / SW_RING) & 1u, abort_addr, WT_SCALES);
                if (!dead) {
                    const uint2 t2 = *reinterpret_cast<const uint2*>(sm + SW_OFF + ((it & (SW_RING - 1)) * T_TILE + token) * 8);
                    ts.below = t2.x; ts.e_g = t2.y;
                    off = (float)((int)ts.e_g - 127 + T_P_SHIFT);
                    dead = !mbar_wait_lean(bar(B_SREADY + b), (it >> 1) & 1u, abort_addr, WT_SREADY);
                }
                if (!dead) {
                    tc_fence_after();
                    load_scores();
                    if (MAXL && ts.e_g != 0u) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) xm[i] = fmaxf(xm[i], __uint_as_float(z[i]));
                    }
                    grow = exponents() > T_TAU + (float)T_P_SHIFT && ts.e_g != 0u;
                    grow |= (((ts.below | 0x80808080u) - shift) & 0x80808080u) != 0x80808080u;     // some byte is smaller
                }
                // Some weight of the 32 heads has outgrown the running maximum, or a block's scale the shift of its weights (or a
                // wait gave up): rare after the first tiles of a request, so only then the maxima over the tokens and the shifts
                // are taken, exchanged and the accumulator rescaled.
                if (named_bar_or(1 + half, 128, grow || dead || *abort_flag != 0)) {
                    if (*abort_flag != 0) dead = true;
                    float mine = -INFINITY;
                    if (!dead) {
                        load_scores();
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            const float r = lanes_max(ts.e_g != 0u ? fmaf(__uint_as_float(z[i]), c, off - (float)T_P_SHIFT) : -INFINITY);
                            if (lane == i) mine = r;
                        }
                        xx[quarter * T_HEADS + hl] = mine;
                        uint32_t low = ts.below;
#pragma unroll
                        for (int o = 16; o >= 1; o >>= 1) low = __vminu4(low, __shfl_xor_sync(0xffffffffu, low, o));
                        kx[half * 4 + quarter] = low;
                        if (j > 0) dead = !mbar_wait_lean(bar(B_PVDONE), (it - 1) & 1u, abort_addr, WT_PVDONE);
                    }
                    const float m_old = -nm[hl];
                    if (named_bar_or(1 + half, 128, dead || *abort_flag != 0)) { dead = true; break; }
                    const float mx = fmaxf(fmaxf(xx[hl], xx[T_HEADS + hl]), fmaxf(xx[2 * T_HEADS + hl], xx[3 * T_HEADS + hl]));
                    const bool up = mx > m_old + T_TAU;    // false while the head has seen no entry
                    const float alpha = up ? ex2(m_old - mx) : 1.f;       // 0 for the first entries
                    if (up) nm[hl] = -mx;                  // the four warps of the head write the same value
                    const uint32_t* kh = kx + half * 4;
                    const uint32_t low = __vminu4(shift, __vminu4(__vminu4(kh[0], kh[1]), __vminu4(kh[2], kh[3])));
                    const uint32_t drop = shift - low;     // (no borrows)
                    shift = low;
                    tc_fence_after();
                    if (__any_sync(0xffffffffu, up) || drop != 0u) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            float a, d;
                            unpack_f32x2(l2[i], a, d);
                            l2[i] = pack_f32x2(a * __shfl_sync(0xffffffffu, alpha, 2 * i), d * __shfl_sync(0xffffffffu, alpha, 2 * i + 1));
                        }
                        if (j > 0) {
#pragma unroll 1
                            for (int bb = 0; bb < 4; ++bb) {
                                const float alpha_b = alpha * __uint_as_float((127u - ((drop >> (8 * bb)) & 0xffu)) << 23);
#pragma unroll
                                for (int hh = 0; hh < 2; ++hh) {
                                    uint32_t o[16];
                                    tmem_ld16(lane_addr + TM_O + 64 * bb + 32 * half + 16 * hh, o);
                                    tmem_wait_ld();
#pragma unroll
                                    for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * __shfl_sync(0xffffffffu, alpha_b, 16 * hh + i));
                                    tmem_st16(lane_addr + TM_O + 64 * bb + 32 * half + 16 * hh, o);
                                }
                            }
                            tmem_wait_st();
                        }
                    }
                    named_bar_sync(1 + half, 128);         // xx is free again, the new maxima are in place
                    load_scores();
                    exponents();
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(B_SFREE + b));      // the score buffer may be overwritten
                const float is = ts.e_g != 0u ? __uint_as_float((254u - ts.e_g) << 23) : 0.f;      // 1 / the group's scale
                const uint64_t is2 = pack_f32x2(is, is);
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    const float p0 = ex2(__uint_as_float(z[i])), p1 = ex2(__uint_as_float(z[i + 1]));
                    fma_f32x2(l2[i / 2], pack_f32x2(p0, p1), is2);
                    z[i] = __float_as_uint(p0); z[i + 1] = __float_as_uint(p1);
                }
                if (it > 0 && !dead) dead = !mbar_wait_lean(bar(B_PVDONE), (it - 1) & 1u, abort_addr, WT_PVDONE);   // the weights of the last tile have been read
                if (dead) continue;
                const uint32_t under = ts.below - shift;   // (no borrows: the shifts are the smallest so far)
#pragma unroll
                for (int bb = 0; bb < 4; ++bb) {           // the weights of dims block bb
                    const float r = __uint_as_float((127u - ((under >> (8 * bb)) & 0xffu)) << 23);
                    uint32_t w8[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        w8[i] = pack_e4m3x4(__uint_as_float(z[4 * i]) * r, __uint_as_float(z[4 * i + 1]) * r, __uint_as_float(z[4 * i + 2]) * r,
                                            __uint_as_float(z[4 * i + 3]) * r);
                    uint8_t* pb = sm + P_OFF + bb * P_BYTES;
                    *reinterpret_cast<uint4*>(pb + swz64((uint32_t)token, (uint32_t)(2 * half))) = make_uint4(w8[0], w8[1], w8[2], w8[3]);
                    *reinterpret_cast<uint4*>(pb + swz64((uint32_t)token, (uint32_t)(2 * half + 1))) = make_uint4(w8[4], w8[5], w8[6], w8[7]);
                }
                fence_proxy_async();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(B_PREADY));
            }
            if (dead) continue;
            // sums over the warp's tokens: halve the list at every exchange, lane i ends with head i
            float s[32];
#pragma unroll
            for (int i = 0; i < 16; ++i) unpack_f32x2(l2[i], s[2 * i], s[2 * i + 1]);
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) {
#pragma unroll
                for (int i = 0; i < o; ++i) {
                    const bool up = (lane & o) != 0;
                    const float send = up ? s[i] : s[i + o], keep = up ? s[i + o] : s[i];
                    s[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
            prev_l = s[0];
            if (MAXL) {
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const float r = lanes_max(xm[i]);
                    if (lane == i) prev_x = r * c;
                }
            }
            prev_m = -nm[hl];
            prev_shift = shift;
            const bool at_begin = tiles.req == meta.begin_req;
            prev = true; prev_req = tiles.req;
            prev_no_split = !p.force_partial && !(at_begin ? meta.first_split : prev_req == meta.end_req ? meta.last_split : 0);
            prev_split = (p.num_splits ? p.num_splits[prev_req] : 0) + (at_begin ? meta.begin_split : 0);
        }
    } else if (warp < T_SCALE) {
        // =================================================================== rows -> K stages (TMA gather)
        // The lanes read the rows' numbers ahead and hand them to the lane that issues the copies through shared memory (by shuffles, under
        // an election for every four rows, the copies took three times the instructions).
        const int quarter = warp - T_PROD;
        int* mine = reinterpret_cast<int*>(sm + IDX_OFF) + 32 * quarter;
        Walk tiles(p, first, step, last);
        bool ok = true;
        int idx = 0;
        uint32_t it = 0;
        for (bool have = true, warm = false; have; warm = true) {
            mine[lane] = idx >= 0 ? idx : NO_ROW;
            have = tiles.next_tile(p, meta);
            idx = have ? tiles.row_index(p, quarter * 32 + lane) : -1;     // read ahead of its use
            if (!warm) continue;
            const uint32_t st = it % NSTAGE;
            if (it >= NSTAGE) ok = mbar_wait_lean(bar(B_KFREE + 4 * st + quarter), ((it / NSTAGE) - 1) & 1u, abort_addr, WT_KFREE);
            if (!ok) break;
            __syncwarp();
            if (elect_one()) {
                uint32_t dst = base + K_OFF + st * K_STAGE + quarter * (32 * 128);
                const uint32_t full = bar(B_KFULL + st);
                mbar_arrive_expect_tx(full, 4 * 32 * 128);
#pragma unroll 1
                for (int q = 0; q < 32; q += 4, dst += 512) {
                    const int4 r = *reinterpret_cast<const int4*>(mine + q);
#pragma unroll
                    for (int b = 0; b < 4; ++b) tma_gather4(dst + b * K_CHUNK, &kv_map, 32 * b, r.x, r.y, r.z, r.w, full);
                }
            }
            __syncwarp();
            // the RoPE stage is free when the scores of the tile before are done
            if (it >= 1) ok = mbar_wait_lean(bar(B_SREADY + ((it - 1) & 1u)), ((it - 1) >> 1) & 1u, abort_addr, WT_SREADY);
            if (!ok) break;
            if (elect_one()) {
                uint32_t dst = base + R_OFF + quarter * (32 * 128);
                mbar_arrive_expect_tx(bar(B_RFULL), 32 * 128);
#pragma unroll 1
                for (int q = 0; q < 32; q += 4, dst += 512) {
                    const int4 r = *reinterpret_cast<const int4*>(mine + q);
                    tma_gather4(dst, &kv_map, ROPE_OFF / 4, r.x, r.y, r.z, r.w, bar(B_RFULL));
                }
            }
            __syncwarp();
            ++it;
        }
    } else if (warp < T_QK) {
        // =================================================================== scale words
        // A warp reads the scales of 32 tokens, makes their words and passes them to the others: row r's word belongs into column r / 32 of
        // lane r % 32, in all four lane quarters, and a warp reaches one of them.  The rows' numbers are read two tiles ahead, their
        // scales one.
        const int quarter = warp - T_SCALE;
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
        uint32_t* words = reinterpret_cast<uint32_t*>(sm + WORD_OFF);
        Walk tiles(p, first, step, last);
        bool ok = true, have = true, have1 = false, have2 = false;     // is there a tile whose rows, scales, words are next
        int idx = -1;
        bool there = false;
        uint4 sc = make_uint4(0u, 0u, 0u, 0u);
        for (uint32_t it = 0, primed = 0; ok && (have || have1 || have2); ) {
            if (primed >= 2 && have2) {
                auto bits = [](uint32_t v) { return max(v, MIN_SCALE_BITS) << 1; };             // the exponent is the upper byte
                const uint32_t lo = __byte_perm(bits(sc.x), bits(sc.y), 0x0073), hi = __byte_perm(bits(sc.z), bits(sc.w), 0x0073);
                const uint32_t mine = there ? __byte_perm(lo, hi, 0x5410) : 0u;
                words[(it & 1u) * T_TILE + quarter * 32 + lane] = there ? mine : 0x7f7f7f7fu;
                uint32_t e_g = max(max(mine & 0xffu, (mine >> 8) & 0xffu), max((mine >> 16) & 0xffu, mine >> 24));
                e_g = max(e_g, __shfl_xor_sync(0xffffffffu, e_g, 4));
                e_g = max(e_g, __shfl_xor_sync(0xffffffffu, e_g, 2));
                e_g = max(e_g, __shfl_xor_sync(0xffffffffu, e_g, 1));
                uint2 ts = make_uint2(NO_SHIFT * 0x01010101u, 0u);
                if (mine != 0u) {
                    ts = make_uint2(e_g * 0x01010101u - mine, e_g);
                    if ((ts.x & 0x80808080u) != 0u) ts.x = __vminu4(ts.x, NO_SHIFT * 0x01010101u);
                }
                if (it >= 2) ok = mbar_wait_lean(bar(B_SREADY + (it & 1u)), ((it >> 1) - 1) & 1u, abort_addr, WT_SREADY);   // the scores two tiles ago are done
                if (named_bar_or(4, 128, !ok)) break;
                uint32_t mx[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) mx[k] = words[(it & 1u) * T_TILE + 32 * k + lane];
                tc_fence_after();
                tmem_st4(lane_addr + TM_SFA + 4 * (it & 1u), mx);
                *reinterpret_cast<uint2*>(sm + SW_OFF + ((it & (SW_RING - 1)) * T_TILE + quarter * 32 + lane) * 8) = ts;
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(B_SCALES + (it & (SW_RING - 1))));
                ++it;
            }
            there = idx >= 0;
            if (there) sc = ld_in(reinterpret_cast<const uint4*>(p.kv + (size_t)idx * ROW_BYTES + SCALE_OFF));
            have2 = have1;
            have1 = have = have && tiles.next_tile(p, meta);
            idx = have ? tiles.row_index(p, quarter * 32 + lane) : -1;
            if (primed < 2) ++primed;
        }
    } else if (warp == T_QK) {
        // =================================================================== score MMAs
        const uint32_t q_lo = desc_lo(base + Q_OFF, 16), qr_lo = desc_lo(base + QR_OFF, 16), r_lo = desc_lo(base + R_OFF, 16);
        Walk tiles(p, first, step, last);
        uint32_t it = 0, rq = 0;
        bool ok = true;
        while (ok && tiles.next_request(p, meta)) {
            ok = mbar_wait_lean(bar(B_QREADY), rq & 1u, abort_addr, WT_QREADY);
            ++rq;
            for (int j = 0; j < tiles.nst && ok; ++j, ++it) {
                const uint32_t st = it % NSTAGE, b = it & 1u;
                if (it >= 2) ok = mbar_wait_lean(bar(B_SFREE + b), ((it >> 1) - 1) & 1u, abort_addr, WT_SFREE);
                if (ok) ok = mbar_wait_lean(bar(B_SCALES + (it & (SW_RING - 1))), (it / SW_RING) & 1u, abort_addr, WT_SCALES);
                if (ok) ok = mbar_wait_lean(bar(B_KFULL + st), (it / NSTAGE) & 1u, abort_addr, WT_KFULL);
                if (!ok) break;
                tc_fence_after();
                const uint32_t k_lo = desc_lo(base + K_OFF + st * K_STAGE, 16), d = tmem + TM_S + 64 * b;
                if (elect_one()) {
#pragma unroll 1
                    for (int bb = 0; bb < 4; ++bb) {
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            mma_mxf8(d, make_desc(k_lo + ((bb * K_CHUNK + k * 32) >> 4), HI_128), make_desc(q_lo + ((bb * Q_CHUNK + k * 32) >> 4), HI_128),
                                     idesc_mx(bb), tmem + TM_SFA + 4 * b, tmem + TM_SFB, (bb | k) != 0);
                    }
                }
                __syncwarp();
                ok = mbar_wait_lean(bar(B_RFULL), it & 1u, abort_addr, WT_RFULL);
                if (!ok) break;
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        mma_f16(d, make_desc(r_lo + ((k * 32) >> 4), HI_128), make_desc(qr_lo + ((k * 32) >> 4), HI_128), IDESC_ROPE, true);
                    tc_commit(bar(B_SREADY + b));
                }
                __syncwarp();
            }
        }
    } else if (warp == T_PV) {
        // =================================================================== P.V MMAs
        Walk tiles(p, first, step, last);
        const uint32_t p_lo = desc_lo(base + P_OFF, 16);
        uint32_t it = 0;
        bool ok = true;
        while (ok && tiles.next_request(p, meta)) {
            for (int j = 0; j < tiles.nst && ok; ++j, ++it) {
                const uint32_t st = it % NSTAGE;
                ok = mbar_wait_lean(bar(B_PREADY), it & 1u, abort_addr, WT_PREADY);
                if (!ok) break;
                tc_fence_after();
                const uint32_t v_lo = desc_lo(base + K_OFF + st * K_STAGE, 16);
                if (elect_one()) {
#pragma unroll 1
                    for (int k = 0; k < 4; ++k) {          // 32 tokens: their rows may be overwritten as soon as they have been read
#pragma unroll
                        for (int b = 0; b < 4; ++b)
                            mma_f8(tmem + TM_O + 64 * b, make_desc(v_lo + ((b * K_CHUNK + k * 4096) >> 4), HI_128),
                                   make_desc(p_lo + ((b * P_BYTES + k * 2048) >> 4), HI_P), IDESC_PV, (j | k) != 0);
                        tc_commit(bar(B_KFREE + 4 * st + k));
                    }
                    tc_commit(bar(B_PVDONE));
                }
                __syncwarp();
            }
        }
    }

    if (*abort_flag != 0) {        // a wait gave up: copies and MMAs may still be in flight; give them time to finish
        const long long t0 = clock64();
        while (clock64() - t0 < 200000) { }
    }
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && *abort_flag != 0 && p.status != nullptr) {
        atomicCAS(p.status, 0, *abort_flag);
        atomicAdd(p.status + 1, 1);
        p.status[2] = blockIdx.x;
    }
    if (warp == T_QK) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

}  // namespace

// Whole requests that each get a pair of SMs to themselves take as long as one request does, and two CTAs walk a long list
// faster than one (attn_duo.cu).  us of this kernel / of attn_duo_kernel, rows in HBM:
//   with maximum logits, 64 heads   8 requests of 256 entries 12.8 / 10.5, 512: 17.3 / 13.5, 1024: 26.0 / 19.2, 2048: 43.6 / 30.0;
//                                   74 of 128: 10.7 / 10.4, 512: 18.5 / 15.0, 2048: 47.1 / 33.0
//                        16 heads   8 of 256 10.3 / 9.9, 1024: 22.6 / 18.5, 2048: 38.5 / 29.3; 74 of 256 11.1 / 11.5, 512: 15.1 / 14.5
//   without them, 64 heads          74 of 128 10.3 / 10.4, 512: 17.7 / 15.0, 768: 22.3 / 17.9
// So the line could lie lower.  It lies where two CTAs took these calls already, because shorter lists would lose something: here the
// weights carry the scale of every block of 128 dims, there a block of V far below its group's scale is shifted into e4m3's subnormals.
// With more requests than pairs of SMs two CTAs need another round: 80 requests of 2048 entries took 51 here and 87 there.
static bool duo_is_faster(const AttnParams& p) {
    if (p.sched != nullptr || p.uniform_k > 1 || p.num_tokens > smla_num_sms() / 2) return false;
    const int blocks = (p.topk + BLOCK_N - 1) / BLOCK_N;
    if (p.num_heads > 32) return blocks >= (p.out_max_logits != nullptr ? 8 : 12);
    return p.out_max_logits != nullptr && blocks >= 16;
}

// One linear array of 656-byte rows (pages without padding between them) and one CTA's worth of heads.
bool attn_tile_takes(const AttnParams& p) {
    return !duo_is_faster(p) && p.num_heads <= T_HEADS && one_linear_array(p);
}

int launch_attn_tile(const AttnParams& p, cudaStream_t stream) {
    if (p.num_tokens == 0) return 0;
    static std::atomic<bool> attr_set[64];
    static int sm_count[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return set_error(SMLA_E_SHAPE, "attn_tile_kernel: device ordinal %d not supported", dev);
    if (!attr_set[dev]) {
        cudaFuncAttributes fa[2];
        if (cudaFuncGetAttributes(&fa[0], attn_tile_kernel<false>) != cudaSuccess || cudaFuncGetAttributes(&fa[1], attn_tile_kernel<true>) != cudaSuccess ||
            fa[0].numRegs != T_REGS_LAUNCH || fa[1].numRegs != T_REGS_LAUNCH)
            return set_error(SMLA_E_DEVICE, "attn_tile_kernel: compiled with %d and %d registers per thread, the warpgroup budgets assume %d",
                             fa[0].numRegs, fa[1].numRegs, T_REGS_LAUNCH);
        cudaError_t e = cudaFuncSetAttribute(attn_tile_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T_SMEM);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(attn_tile_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T_SMEM);
        if (e != cudaSuccess) return set_error((int)e, "attn_tile_kernel: cannot reserve %u bytes of shared memory: %s", T_SMEM, cudaGetErrorString(e));
        cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev);
        attr_set[dev] = true;
    }
    CUtensorMap map;
    if (int e = rows_tensor_map(p.kv, &map)) return e;
    const int parts = p.sched ? p.num_parts : p.uniform_k > 1 ? p.uniform_k * p.num_tokens : (p.num_tokens < sm_count[dev] ? p.num_tokens : sm_count[dev]);
    const dim3 grid(parts);
    auto* kernel = p.out_max_logits != nullptr ? attn_tile_kernel<true> : attn_tile_kernel<false>;
    launch_dependent(kernel, grid, dim3(T_THREADS), T_SMEM, stream, p, map);
    return check_launch("attn_tile_kernel");
}

}  // namespace smla

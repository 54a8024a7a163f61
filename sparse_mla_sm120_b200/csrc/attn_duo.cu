// Sparse-MLA attention of 65 to 128 query heads over packed 656-byte rows (sm_100a): whole requests and equal partitions of them on
// a pair of SMs, rows gathered by TMA straight into the operands of the MMAs.
//
// Work unit.  As in attn_pair.cu a cluster of two CTAs owns every parts-th whole request (or one of the equal partitions of a request), CTA r
// holds half of the heads and every MMA is a tcgen05.mma.cta_group::2 with M = 128 (64 heads of each CTA):
//   * Q.K^T: B = the 64 rows of a 128-token tile that each CTA has gathered, N = 128 tokens.
//   * P.V:   B = V^T, N = 256 dims of an MMA, 128 from each CTA: CTA r supplies dims [256 r, +256) of all 128 tokens.
// What is different is where the operands come from.  There a row goes through a raw slot and the registers of a gather
// warp (exponent shift) into the K stage, and from there by shared-memory copies into the V slots of both CTAs: three
// coupled chains.  Here K and V are gathered apart by TMA gather4 (a CTA's own rows whole for K, all rows' 256 dims for V: 72 KB per
// tile and CTA instead of 41 KB, which the L2 has to spare), nothing waits for a copy of anything else, and the four
// scales of a row are applied by the tensor core to K (kind::mxf8f6f4, one power of two per row and 32 values).
// V's scale is a factor of the token and cannot be applied by P.V; its bytes are brought onto one scale per group of eight
// tokens (the largest of their 4 x 8), in place and only the 128-byte pieces that have another one.
// Numerics are those of attn_pair.cu (the same groups, the same weights), with K exact instead of shifted.
//
// What bounds it is the issue of instructions (ncu, 740 tokens of 2048 entries, rows in L2): 8650 per tile and CTA on 32 warps, request
// switches included, issue slots 72 % busy, the ALU pipe 61 %, the tensor pipe 38 %.  The copies of a tile alone would need 1750 cycles
// (TMA gather4 moves a row's 128 bytes in 3 cycles, whatever the order), the MMAs 1150; the first version of the kernel, of 9500
// instructions, took 2650 (clock64), the pair kernel 4000.  Hence the manner of the code: loops instead of unrolled copies, one place in
// the code for what is done at several times, walkers and waits of few instructions (at 104 KB of code the instruction cache hit 64 %
// and the kernel was slower than the pair kernel, now 96 %), and shifts of V spread over eight warps, since LOP3 and PRMT go out every
// other cycle only.
// A long run is held at 1640 MHz by the power limit (the pair kernel: 1905 MHz), which takes back some of the gain:
// 4096 tokens of top-k 2048 2230 -> 1815 us in a row (the first version, of 9500 instructions per tile: 1930, and 1620 alone where the
// pair kernel takes 2170); 64 requests 49.2 -> 43.4 us, two tokens of 64 requests 96.8 -> 83.8 us.
// Measured and not kept: Q and the epilogue on the softmax warps as in attn_pair.cu (15000 cycles between two requests, now 4000);
// five V slots with a warp of its own each (a warp shifts half a tile in 6500 cycles), V warps that copy and shift (the copies wait for
// the shifts), K and V copied by the same warps (they are the limit then), rows asked into L2 a tile ahead (no gain, 3 % lost with two
// tokens per request), sleeping waits and a poller per group of warps (a suspended wait costs no issue slots).
//
// Warp roles (1024 threads per CTA):
//   warps 0-7    softmax (thread = one head x 32 tokens of a tile), as in attn_pair.cu
//   warps 8-11   scales: the scale words of all 128 tokens into tensor memory and into records in shared memory; epilogue
//   warps 12-15  q of the next request; epilogue
//   warps 16-17  gather K, warps 18, 19, 22 and 23 gather V
//   warp 20      even CTA: issues the score MMAs; odd CTA: passes on that its K rows have landed
//   warp 21      issues the P.V MMAs (even CTA)
//   warps 24-31  V: shift the pieces whose scale is not the group's
// Every wait is bounded; a wait that gives up records a code in status[] and the CTA drains and exits.  Warps that meet at a
// named barrier leave the loop together.
#include "attn_common.cuh"
#include "rows_map.cuh"
#include "sm100_ptx.cuh"

namespace smla {

namespace {

using namespace ptx;
using namespace attn;

constexpr int N_SM_WARPS = 8, SCALE_WARP0 = 8, QUANT_WARP0 = 12, COPY_WARP0 = 16, V_WARP0 = 18, QK_WARP = 20, PV_WARP = 21, FIX_WARP0 = 24;
constexpr int N_FIX_WARPS = 8, N_AUX_WARPS = COPY_WARP0 - SCALE_WARP0;
constexpr int DUO_THREADS = 32 * 32;
constexpr int REGS_LAUNCH = 64, REGS_SOFTMAX = 88, REGS_AUX = 80, REGS_COPY = 40, REGS_FIX = 48;
static_assert((N_SM_WARPS * REGS_SOFTMAX + N_AUX_WARPS * REGS_AUX + 8 * REGS_COPY + N_FIX_WARPS * REGS_FIX) * 32 <= DUO_THREADS * REGS_LAUNCH, "register budgets exceed what the CTA owns");

constexpr int OWN_N = 64;                // rows of K that each CTA gathers of a tile
constexpr int P_SHIFT = 5;               // P' is stored as e4m3(P' * 2^P_SHIFT)
constexpr float RESCALE_TAU = 3.0f;      // lazy-rescale threshold (log2 units); P' <= 2^TAU
constexpr int NST = 2;                   // K stages, score buffers and P' buffers follow the tile's parity
constexpr int NVS = 4;                   // V slots of half a tile each: two per half
constexpr int HALF_N = 64;

constexpr uint32_t CHUNK = OWN_N * 128;              // 128 dims (or the RoPE) of 64 rows, K-major 128B swizzle
constexpr uint32_t Q_OFF = 0;                        // q e4m3, four chunks of [64 heads x 128 dims]
constexpr uint32_t QR_OFF = Q_OFF + 4 * CHUNK;       // q RoPE bf16
constexpr uint32_t PB_OFF = QR_OFF + CHUNK;          // P' e4m3 [64 heads x 128 tokens], two buffers
constexpr uint32_t KS_OFF = PB_OFF + NST * CHUNK;    // K stages: four chunks and the RoPE
constexpr uint32_t KS_BYTES = 5 * CHUNK;
constexpr uint32_t VS_OFF = KS_OFF + NST * KS_BYTES; // V slots: two blocks of [64 tokens x 128 dims], MN-major 128B swizzle
constexpr uint32_t V_BLOCK = HALF_N * 128, VS_BYTES = 2 * V_BLOCK, V_STEP = 32 * 128;
constexpr int REC_RING = 8;                          // records outlive their K stage
constexpr uint32_t REC_OFF = VS_OFF + NVS * VS_BYTES;         // per token: by how many powers of two its four blocks lie below the group's scale, four bits each
constexpr uint32_t GRP_OFF = REC_OFF + REC_RING * TILE_N * 2; // per group of eight tokens: exponent of its scale | valid bits << 8
constexpr uint32_t GRP_BYTES = TILE_N / 8 * 4;
constexpr uint32_t IDX_OFF = GRP_OFF + REC_RING * GRP_BYTES;  // the rows that a gathering warp is about to ask for, 32 each
constexpr uint32_t FIX_OFF = IDX_OFF + 6 * 32 * 4;      // the V pieces that a warp is about to shift
constexpr uint32_t FIX_LIST = 48;
constexpr uint32_t WORD_OFF = FIX_OFF + N_FIX_WARPS * FIX_LIST * 4;    // the rows' scale words on their way to tensor memory: [2][128]
constexpr uint32_t XCH_OFF = WORD_OFF + 2 * TILE_N * 4;       // row-maximum exchange [4][64] fp32
constexpr int REQ_RING = 4;                                   // requests that the roles may be apart
constexpr uint32_t SQ_OFF = XCH_OFF + 4 * 64 * 4;             // exponents of the heads' q scales, [REQ_RING][64] bytes
constexpr uint32_t SUM_OFF = SQ_OFF + REQ_RING * 64;          // a finished request's sums: [2] x ([4][64] denominators, [4][64] maxima, [64] m)
constexpr uint32_t SUM_BYTES = 9 * 64 * 4;
constexpr uint32_t B_OFF = SUM_OFF + 2 * SUM_BYTES;
// Barriers.  "P" barriers collect arrivals from both CTAs and are used in the even CTA only.
constexpr int B_KFULL = 0, B_KPEERP = B_KFULL + NST, B_VFULL = B_KPEERP + NST, B_VREADYP = B_VFULL + NVS, B_VFREE = B_VREADYP + NVS,
              B_SCALES = B_VFREE + NVS, B_SCALEP = B_SCALES + REC_RING, B_SREADY = B_SCALEP + NST, B_SFREEP = B_SREADY + NST,
              B_PREADYP = B_SFREEP + NST, B_PVDONE = B_PREADYP + NST, B_QREADYP = B_PVDONE + NST, B_QSCALE = B_QREADYP + 1,
              B_SUMS = B_QSCALE + REQ_RING, B_SUMFREE = B_SUMS + 2, B_OFREEP = B_SUMFREE + 2, B_QFREE = B_OFREEP + 1, B_QPART = B_QFREE + 1, B_N = B_QPART + 4;
constexpr uint32_t MISC_OFF = B_OFF + B_N * 8;       // tmem base (4 B), abort flag (4 B)
constexpr uint32_t SMEM_ALLOC = MISC_OFF + 16 + 1024;
static_assert(SMEM_ALLOC <= 227 * 1024, "shared memory budget");
static_assert(QR_OFF == Q_OFF + 4 * CHUNK && KS_BYTES == 5 * CHUNK, "the RoPE follows the four chunks");
static_assert(KS_OFF % 1024 == 0 && VS_OFF % 1024 == 0 && KS_BYTES % 1024 == 0 && GRP_OFF % 16 == 0 && B_OFF % 8 == 0, "alignment");

// tensor memory: O 256 columns, two score buffers of 64, scale words (the heads': all 1; the tokens': four columns per buffer), the
// next request's quantised q on its way to shared memory (64 columns of no-PE values, 16 of RoPE)
constexpr uint32_t TMEM_COLS = 512, TM_O = 0, TM_S = 256, TM_SFA = 384, TM_SFB = 388, TM_Q = 400, TM_QR = 464;
// kind::mxf8f6f4: scale type UE8M0 (bit 23), the byte of the scale words that B uses (bits 4-5), M >> 7 (bits 27-28)
__host__ __device__ constexpr uint32_t idesc_mx(uint32_t b_byte) {
    return (b_byte << 4) | (FMT_E4M3 << 7) | (FMT_E4M3 << 10) | ((TILE_N >> 3) << 17) | (1u << 23) | ((128u >> 7) << 27);
}
constexpr uint32_t IDESC_ROPE = instr_desc(FMT_BF16, FMT_BF16, false, false, 128, TILE_N);
constexpr uint32_t IDESC_PV = instr_desc(FMT_E4M3, FMT_E4M3, false, true, 128, 256);
constexpr uint32_t HI_128 = desc_hi(1024, (uint32_t)SWIZZLE_128B);

// Named barriers: softmax warps of 32 heads (two), the warps that share the first q, those that hand over the scales.
enum { NB_SOFTMAX = 1, NB_FIRST_Q = 4, NB_SCALE = 5 };

// give-up codes reported through status[0]
enum { WD_KFULL = 71, WD_KPEER = 72, WD_VFULL = 73, WD_VREADY = 74, WD_SCALES = 75, WD_SREADY = 76, WD_SFREE = 77, WD_PREADY = 78, WD_PVDONE = 79, WD_QREADY = 80,
       WD_QSCALE = 81, WD_SUMS = 82, WD_OFREE = 83, WD_QFREE = 84, WD_VFREE = 85, WD_SUMFREE = 86, WD_QPART = 87 };

__device__ __forceinline__ uint32_t swz(uint32_t row, uint32_t piece) { return row * 128u + ((piece ^ (row & 7u)) << 4); }

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(DUO_THREADS, 1) attn_duo_kernel(const AttnParams p, const __grid_constant__ CUtensorMap kv_map) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* sm = smem_raw + (base - raw);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + MISC_OFF + 4);
    const uint32_t abort_addr = base + MISC_OFF + 4;
    auto bar = [&](int i) -> uint32_t { return base + B_OFF + 8u * i; };
    auto barp = [&](int i) -> uint32_t { return mapa_shared(bar(i), 0); };   // the even CTA's copy of barrier i

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_ctarank();          // 0: the CTA that issues the MMAs
    const int part = blockIdx.x >> 1;
    const int heads_cta = (p.num_heads + 1) >> 1;     // heads per CTA
    const int head0 = (int)rank * heads_cta;
    const int live_heads = min(heads_cta, max(p.num_heads - head0, 0));

    if (tid == 0) {
        for (int s = 0; s < NST; ++s) {
            mbar_init(bar(B_KFULL + s), 2);          // + the bytes of this CTA's rows
            mbar_init(bar(B_KPEERP + s), 1);                 // the odd CTA's rows have landed
            mbar_init(bar(B_SCALEP + s), 2 * 4);
            mbar_init(bar(B_SREADY + s), 1 + 4);             // the scores are done (and so the K stage is free), the records of their scales are in place
            mbar_init(bar(B_SFREEP + s), 2 * N_SM_WARPS);
            mbar_init(bar(B_PREADYP + s), 2 * N_SM_WARPS);
            mbar_init(bar(B_PVDONE + s), 1);
            mbar_init(bar(B_SUMS + s), N_SM_WARPS);          // a finished request's sums are in shared memory
            mbar_init(bar(B_SUMFREE + s), N_AUX_WARPS);
        }
        for (int s = 0; s < NVS; ++s) {
            mbar_init(bar(B_VFULL + s), 2);                  // + the bytes of the half tile's 256 dims
            mbar_init(bar(B_VREADYP + s), 2 * N_FIX_WARPS / 2);
            mbar_init(bar(B_VFREE + s), 1);
        }
        for (int s = 0; s < REC_RING; ++s) mbar_init(bar(B_SCALES + s), 4);
        for (int s = 0; s < REQ_RING; ++s) mbar_init(bar(B_QSCALE + s), 4);
        for (int s = 0; s < 4; ++s) mbar_init(bar(B_QPART + s), 1);      // the scaler's part of a lane quarter's q is in tensor memory
        mbar_init(bar(B_QREADYP), 2 * 4);
        mbar_init(bar(B_QFREE), 1);                          // the last scores of a request are done
        mbar_init(bar(B_OFREEP), 2 * N_AUX_WARPS);           // a finished request's accumulator has been read
        *abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == QK_WARP) {
        tmem_alloc_pair(base + MISC_OFF, TMEM_COLS);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();          // the partner's barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(sm + MISC_OFF);

    // Everything above needs nothing from the kernels before this one, and the one after it may start its own prologue.
    grid_dep_wait();
    grid_dep_launch();
    SchedMeta meta;
    int first, step, last;
    if (p.uniform_k > 1) {
        meta = load_meta(p, part);
        first = meta.begin_req; step = 1; last = min(meta.end_req, p.num_tokens - 1);
    } else {                                          // whole requests; neighbours differ little in length, so every pair takes each parts-th
        meta.begin_block = 0; meta.end_block = 0x7fffffff;
        meta.begin_split = 0; meta.first_split = meta.last_split = 0; meta.pad = 0;
        first = part; step = (int)(gridDim.x >> 1); last = p.num_tokens - 1;
        meta.begin_req = 0; meta.end_req = last;
    }
    // The sign of the softmax scale goes into q, so that scores are always multiplied by a positive number.
    const uint32_t scale_sign = __float_as_uint(p.sm_scale) & 0x80000000u;
    // A lane's 16 of the 512 no-PE dims of a head, quantised to e4m3 with one power of two per head: returns its exponent.
    auto quantise = [&](const uint4& v0, const uint4& v1, uint32_t (&o)[4]) -> uint32_t {
        const uint32_t x[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
        uint32_t am = 0u;                                  // magnitudes of bf16 numbers order as integers do
#pragma unroll
        for (int c = 0; c < 8; ++c) am = __vmaxu2(am, x[c] & 0x7fff7fffu);
        am = __reduce_max_sync(0xffffffffu, max(am & 0xffffu, am >> 16));
        const float sq = pow2_ceil(fmaxf(__uint_as_float(am << 16), 1e-4f) * (1.f / 448.f));
        const float is = __uint_as_float((0x7f000000u - __float_as_uint(sq)) | scale_sign);   // 1/sq, sq a power of two
#pragma unroll
        for (int c = 0; c < 4; ++c)
            o[c] = pack_e4m3x4(bf16lo(x[2 * c]) * is, bf16hi(x[2 * c]) * is, bf16lo(x[2 * c + 1]) * is, bf16hi(x[2 * c + 1]) * is);
        return __float_as_uint(sq) >> 23;
    };
    // 16 bytes of a head's RoPE, divided by its scale
    auto rope = [&](const uint4& v, uint32_t exponent) {
        const __nv_bfloat162 f = __float2bfloat162_rn(__uint_as_float(((254u - exponent) << 23) | scale_sign));
        return make_uint4(mul_bf16x2(v.x, f), mul_bf16x2(v.y, f), mul_bf16x2(v.z, f), mul_bf16x2(v.w, f));
    };
    // The first request's q: there is nothing to overlap it with, so sixteen warps take four heads each, all loads at once.
    if (warp < COPY_WARP0) {
        Walk first_request(p, first, step, last);
        if (first_request.next_request(p, meta)) {
            const __nv_bfloat16* q0 = p.q + ((size_t)first_request.req * p.num_heads + head0) * D_QK;
            uint8_t* sqv = sm + SQ_OFF;
            uint4 v[9];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int h = 4 * warp + k;
                v[2 * k] = v[2 * k + 1] = make_uint4(0, 0, 0, 0);
                if (h < live_heads) {
                    v[2 * k] = ld_in(reinterpret_cast<const uint4*>(q0 + (size_t)h * D_QK + lane * 16));
                    v[2 * k + 1] = ld_in(reinterpret_cast<const uint4*>(q0 + (size_t)h * D_QK + lane * 16 + 8));
                }
            }
            const uint32_t hr = 4 * warp + (lane >> 3);
            v[8] = make_uint4(0, 0, 0, 0);
            if ((int)hr < live_heads) v[8] = ld_in(reinterpret_cast<const uint4*>(q0 + (size_t)hr * D_QK + D_NOPE + (lane & 7) * 8));
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                uint32_t o[4];
                const uint32_t e = quantise(v[2 * k], v[2 * k + 1], o);
                *reinterpret_cast<uint4*>(sm + Q_OFF + (lane >> 3) * CHUNK + swz(4 * warp + k, (uint32_t)lane & 7u)) = make_uint4(o[0], o[1], o[2], o[3]);
                if (lane == 0) sqv[4 * warp + k] = (uint8_t)e;
            }
            __syncwarp();
            *reinterpret_cast<uint4*>(sm + QR_OFF + swz(hr, (uint32_t)lane & 7u)) = rope(v[8], sqv[hr]);
            fence_proxy_async();
            named_bar_sync(NB_FIRST_Q, 32 * COPY_WARP0);
        }
    }
    if (warp < N_SM_WARPS) setmaxnreg_inc<REGS_SOFTMAX>();
    else if (warp < COPY_WARP0) setmaxnreg_inc<REGS_AUX>();
    else if (warp < FIX_WARP0) setmaxnreg_dec<REGS_COPY>();
    else setmaxnreg_dec<REGS_FIX>();


    if (warp < N_SM_WARPS) {
        // =================================================================== softmax
        const int quarter = warp & 3, ch = warp >> 2;     // TMEM lane quarter, column half of a score buffer
        const int grp = quarter & 1;                      // warps with equal grp share 32 heads
        const int thalf = quarter >> 1;                   // scores: token half; accumulator: half of the output dims
        const int hrow = grp * 32 + lane;                 // head row inside this CTA
        const bool live = hrow < live_heads;
        const int xpart = thalf * 2 + ch;                 // which of the four partial rows this thread holds
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
        float* xch = reinterpret_cast<float*>(sm + XCH_OFF);   // [4][64]
        Walk tiles(p, first, step, last);
        uint32_t it = 0, rq = 0;                          // tiles and requests of this CTA so far
        bool dead = false;                                // a wait of this warp gave up: no more work, only barriers
        bool stop = false;
        for (; !stop && tiles.next_request(p, meta); ++rq) {
            if (!dead) dead = !mbar_wait_lean(bar(B_QSCALE + (rq & (REQ_RING - 1))), (rq / REQ_RING) & 1u, abort_addr, WD_QSCALE);
            // Never 0: the scores of entries without a row are -inf, and -inf times a softmax scale of 0 would be no number.
            // 2^-62 times any score is far below one step of an exponent.
            const float sq = __uint_as_float((uint32_t)sm[SQ_OFF + (rq & (REQ_RING - 1)) * 64 + hrow] << 23);
            const float my_sqc = live ? fmaxf(sq * fabsf(p.sm_scale) * LOG2E, 0x1p-62f) : 1.f;
            float m_run = -INFINITY;   // running maximum of z (lags by at most RESCALE_TAU)
            float l_run = 0.f;         // this thread's share of the sum of P'/s (scaled by 2^P_SHIFT)
            float x_max = -INFINITY;   // this thread's share of the maximum of the scaled logits (max_logits output)
            for (int j = 0; j < tiles.nst; ++j, ++it) {
                const uint32_t b = it & 1u, ring = it & (REC_RING - 1);
                uint32_t sv[32];                           // raw scores; -inf where there is no entry
                float mx_loc = -INFINITY;
                float off_g[4], inv_g[4];                  // of the four groups of eight tokens that this thread holds: z = s * c + off, 1/s
                const uint8_t* grec = sm + GRP_OFF + ring * GRP_BYTES + (8 * thalf + 4 * ch) * 4;
                if (!dead) dead = !mbar_wait_lean(bar(B_SREADY + b), (it >> 1) & 1u, abort_addr, WD_SREADY);
                if (!dead) {
                    tc_fence_after();
                    tmem_ld32(lane_addr + TM_S + 64 * b + 32 * ch, sv);
                    const uint4 g4 = *reinterpret_cast<const uint4*>(grec);
                    const uint32_t gr[4] = {g4.x, g4.y, g4.z, g4.w};
                    uint32_t valid = 0u;
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        const uint32_t e = gr[g] & 0xffu;
                        off_g[g] = (float)((int)e - 127);
                        inv_g[g] = __uint_as_float((254u - e) << 23);
                        valid |= (gr[g] >> 8) << (8 * g);
                    }
                    tmem_wait_ld();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_remote(barp(B_SFREEP + b));     // the score buffer may be overwritten
                    if (valid != 0xffffffffu) {                                // the same in all lanes
#pragma unroll
                        for (int t = 0; t < 32; ++t)
                            if (!((valid >> t) & 1u)) sv[t] = 0xff800000u;     // no entry: weight exactly 0
                    }
                    float gx = -INFINITY;
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        const uint32_t* v = sv + 8 * g;
                        auto f = [](uint32_t x) { return __uint_as_float(x); };
                        const float gm = fmaxf(fmaxf(fmaxf(f(v[0]), f(v[1])), fmaxf(f(v[2]), f(v[3]))),
                                               fmaxf(fmaxf(f(v[4]), f(v[5])), fmaxf(f(v[6]), f(v[7]))));
                        mx_loc = fmaxf(mx_loc, fmaf(gm, my_sqc, off_g[g]));
                        gx = fmaxf(gx, gm);
                    }
                    x_max = fmaxf(x_max, gx * my_sqc);                         // the scaled logit itself, without log2(s)
                }
                // Some row of the group of 128 threads has outgrown its running maximum (or a wait gave up): rare after the
                // first tiles of a request, so only then the four partial row maxima are exchanged.
                if (named_bar_or(NB_SOFTMAX + grp, 128, mx_loc > m_run + RESCALE_TAU || dead)) {
                    xch[xpart * 64 + hrow] = mx_loc;
                    if (named_bar_or(NB_SOFTMAX + grp, 128, dead || *abort_flag != 0)) { stop = true; break; }
                    const float* xr = xch + hrow;
                    const float mx = fmaxf(fmaxf(xr[0], xr[64]), fmaxf(xr[128], xr[192]));
                    const bool grow = mx > m_run + RESCALE_TAU;   // false while the row has seen no valid entry
                    if (j > 0) {   // the accumulator holds earlier tiles: wait for the last P.V, then scale it
                        dead = !mbar_wait_lean(bar(B_PVDONE + ((it - 1) & 1u)), ((it - 1) >> 1) & 1u, abort_addr, WD_PVDONE);
                        if (dead) continue;
                        tc_fence_after();
                    }
                    const float alpha = grow ? ex2(m_run - mx) : 1.f;   // 2^-inf = 0 for the first tile
                    if (grow) { m_run = mx; l_run *= alpha; }
                    if (j > 0) {
#pragma unroll 1
                        for (int c = 0; c < 128; c += 16) {
                            uint32_t o[16];
                            tmem_ld16(lane_addr + TM_O + 128 * ch + c, o);
                            tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                            tmem_st16(lane_addr + TM_O + 128 * ch + c, o);
                        }
                        tmem_wait_st();
                    }
                }
                const float m_off = ((m_run == -INFINITY) ? 0.f : m_run) - (float)P_SHIFT;
                const uint64_t c2 = pack_f32x2(my_sqc, my_sqc);
                uint32_t pw[8];
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    // two scores per FMA and per addition (packed fp32, each half rounded as the scalar operation)
                    const uint64_t e2 = pack_f32x2(off_g[g] - m_off, off_g[g] - m_off);
                    uint64_t l2 = 0ull;
#pragma unroll
                    for (int t = 8 * g; t < 8 * g + 8; t += 4) {
                        uint64_t a01 = e2, a23 = e2;
                        fma_f32x2(a01, pack_f32x2(__uint_as_float(sv[t + 0]), __uint_as_float(sv[t + 1])), c2);
                        fma_f32x2(a23, pack_f32x2(__uint_as_float(sv[t + 2]), __uint_as_float(sv[t + 3])), c2);
                        float p0, p1, p2, p3;
                        unpack_f32x2(a01, p0, p1); unpack_f32x2(a23, p2, p3);
                        p0 = ex2(p0); p1 = ex2(p1); p2 = ex2(p2); p3 = ex2(p3);
                        add_f32x2(l2, pack_f32x2(p0, p1));
                        add_f32x2(l2, pack_f32x2(p2, p3));
                        pw[t >> 2] = pack_e4m3x4(p0, p1, p2, p3);
                    }
                    float l0, l1;
                    unpack_f32x2(l2, l0, l1);
                    l_run = fmaf(l0 + l1, inv_g[g], l_run);
                }
                // P' of tokens [64*thalf + 32*ch, +32) of head hrow: two 16-byte pieces of the row
                uint8_t* pb = sm + PB_OFF + b * CHUNK;
                *reinterpret_cast<uint4*>(pb + swz(hrow, 4 * thalf + 2 * ch)) = make_uint4(pw[0], pw[1], pw[2], pw[3]);
                *reinterpret_cast<uint4*>(pb + swz(hrow, 4 * thalf + 2 * ch + 1)) = make_uint4(pw[4], pw[5], pw[6], pw[7]);
                fence_proxy_async();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_remote(barp(B_PREADYP + b));
            }
            if (stop || dead) continue;                    // (a warp that is dead meets the others at the next tile's barrier)
            if (rq >= 2) dead = !mbar_wait_lean(bar(B_SUMFREE + (rq & 1u)), ((rq >> 1) - 1) & 1u, abort_addr, WD_SUMFREE);
            if (dead) continue;
            float* sums = reinterpret_cast<float*>(sm + SUM_OFF + (rq & 1u) * SUM_BYTES);
            sums[xpart * 64 + hrow] = l_run;
            sums[256 + xpart * 64 + hrow] = x_max;
            if (xpart == 0) sums[512 + hrow] = m_run;
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(B_SUMS + (rq & 1u)));
        }
    } else if (warp < COPY_WARP0) {
        // =================================================================== scales (warps 8-11), Q (warps 12-15), epilogue (all)
        // The scale words of a tile are handed over two tiles ahead of its scores.  The next request's q is read and quantised while
        // this one's tiles run (a load that has to queue behind the gathers takes 2000 cycles), waits in tensor memory, and goes
        // to shared memory as soon as the last scores of this request are done.  A request's output is written when its last P.V is,
        // under the first scores and weights of the next.
        // Scales: a pair MMA with M = 128 leaves the scores of tokens 0-63 in lanes 0-63 and those of tokens 64-127 in lanes 64-127,
        // and every lane quarter takes the tokens' scale words from its own lanes: column c of lane i of quarter q holds the word
        // of token 64 (q / 2) + 32 c + i; a warp makes the words of tokens 32 q + i and passes them on.  The next tile's scales are asked for when this tile's words have been handed over.
        const bool scaler = warp < QUANT_WARP0;
        const int quarter = warp & 3, ch = scaler ? 0 : 1;
        const int grp = quarter & 1, thalf = quarter >> 1, hrow = grp * 32 + lane, head = head0 + hrow;
        const bool live = hrow < live_heads;
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
        // Heads [i0, i0 + n) of the 16 of a lane quarter into tensor memory
        auto prepare_q = [&](int req, uint32_t r, int i0, int n) {
            const __nv_bfloat16* q0 = p.q + ((size_t)req * p.num_heads + head0) * D_QK;
            uint8_t* sqv = sm + SQ_OFF + (r & (REQ_RING - 1)) * 64;
#pragma unroll 1
            for (int i = i0; i < i0 + n; i += 4) {
                uint4 v[8];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int h = 16 * quarter + i + k;
                    v[2 * k] = v[2 * k + 1] = make_uint4(0, 0, 0, 0);
                    if (h < live_heads) {
                        v[2 * k] = ld_in(reinterpret_cast<const uint4*>(q0 + (size_t)h * D_QK + lane * 16));
                        v[2 * k + 1] = ld_in(reinterpret_cast<const uint4*>(q0 + (size_t)h * D_QK + lane * 16 + 8));
                    }
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    uint32_t o[4];
                    const uint32_t e = quantise(v[2 * k], v[2 * k + 1], o);
                    tmem_st4(lane_addr + TM_Q + 4 * (i + k), o);
                    if (lane == 0) sqv[16 * quarter + i + k] = (uint8_t)e;
                }
            }
            __syncwarp();
#pragma unroll 1
            for (int i = i0; i < i0 + n; i += 8) {
                uint4 v[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const int h = 16 * quarter + i + 4 * k + (lane >> 3);
                    v[k] = make_uint4(0, 0, 0, 0);
                    if (h < live_heads) v[k] = ld_in(reinterpret_cast<const uint4*>(q0 + (size_t)h * D_QK + D_NOPE + (lane & 7) * 8));
                }
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const uint4 t = rope(v[k], sqv[16 * quarter + i + 4 * k + (lane >> 3)]);
                    const uint32_t o[4] = {t.x, t.y, t.z, t.w};
                    tmem_st4(lane_addr + TM_QR + i + 4 * k, o);
                }
            }
            tmem_wait_st();
        };
        bool ok = true;
        Walk ahead(p, first, step, last);                 // the tile whose rows are named next
        uint32_t sit = 0, primed = 0;                     // number of the next tile to hand over; stages of the read-ahead that are filled
        int idx = -1;
        uint4 sc = make_uint4(0u, 0u, 0u, 0u);
        bool there = false;
        uint32_t* words = reinterpret_cast<uint32_t*>(sm + WORD_OFF);
        if (scaler) {
            const uint32_t ones[4] = {0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu, 0x7f7f7f7fu};
            tmem_st4(lane_addr + TM_SFA, ones);           // the heads' scales stay outside the MMAs
        }
        Walk tiles(p, first, step, last);
        uint32_t it = 0, rq = 0;                          // first tile and number of the request
        const bool whole = p.uniform_k <= 1;              // requests are not cut
        bool together = false;                            // the scalers leave because one of them has given up, and all know it
        bool prev = false;
        int prev_req = 0, last_nst = 0;
        while (true) {
            const bool have = tiles.next_request(p, meta);
            if (have && rq > 0) {
                // Behind a short request the scaler takes half of the heads; behind a long one the quantiser has the time, and the
                // scaler, who comes here only when all tiles of that request are handed over, would be late with the next ones.
                const bool shared = last_nst < 8;
                if (scaler && shared) ok = mbar_wait_lean(bar(B_QSCALE + ((rq - 1) & (REQ_RING - 1))), ((rq - 1) / REQ_RING) & 1u, abort_addr, WD_QSCALE);   // the last q has left tensor memory
                if (!ok) break;
                if (!scaler || shared) prepare_q(tiles.req, rq, shared && !scaler ? 8 : 0, shared ? 8 : 16);
                tc_fence_before();
                __syncwarp();
                if (scaler && lane == 0) mbar_arrive(bar(B_QPART + quarter));
            }
            last_nst = tiles.nst;
            const int n = have ? tiles.nst : 1, j_epi = min(1, n - 1);
            for (int j = 0; j < n; ++j) {
                // ---- scales of the next tile (the rows' numbers are read two tiles ahead, their scales one)
                for (bool filling = true; have && scaler && filling; ) {
                    filling = primed < 2;
                    if (!filling) {
                        const uint32_t ring = sit & (REC_RING - 1), b = sit & 1u;
                        auto bits = [](uint32_t v) { return max(v, MIN_SCALE_BITS) << 1; };             // the exponent is the upper byte
                        const uint32_t lo = __byte_perm(bits(sc.x), bits(sc.y), 0x0073), hi = __byte_perm(bits(sc.z), bits(sc.w), 0x0073);
                        const uint32_t mine = there ? __byte_perm(lo, hi, 0x5410) : 0u;
                        words[b * TILE_N + 32 * quarter + lane] = there ? mine : 0x7f7f7f7fu;
                        const uint32_t valid = __ballot_sync(0xffffffffu, there);
                        uint32_t e_g = max(max(max(mine & 0xffu, (mine >> 8) & 0xffu), max((mine >> 16) & 0xffu, mine >> 24)), MIN_SCALE_BITS >> 23);
                        e_g = max(e_g, __shfl_xor_sync(0xffffffffu, e_g, 4));
                        e_g = max(e_g, __shfl_xor_sync(0xffffffffu, e_g, 2));
                        e_g = max(e_g, __shfl_xor_sync(0xffffffffu, e_g, 1));
                        // by how many powers of two each block of the token lies below the group's scale, at most 15: a byte each, then four bits each
                        uint32_t d = mine != 0u ? __vminu4(e_g * 0x01010101u - mine, 0x0f0f0f0fu) : 0u;
                        d |= d >> 4;
                        d = __byte_perm(d, 0u, 0x4420);
                        if (sit >= 2) ok = mbar_wait_lean(bar(B_SREADY + b), ((sit >> 1) - 1) & 1u, abort_addr, WD_SREADY);   // the scores two tiles ago are done
                        together = named_bar_or(NB_SCALE, 128, !ok);
                        if (together) { ok = false; break; }
                        const uint32_t mx[2] = {words[b * TILE_N + 64 * thalf + lane], words[b * TILE_N + 64 * thalf + 32 + lane]};
                        tc_fence_after();
                        tmem_st2(lane_addr + TM_SFB + 4 * b, mx);
                        *reinterpret_cast<uint16_t*>(sm + REC_OFF + (ring * TILE_N + 32 * quarter + lane) * 2) = (uint16_t)d;
                        if ((lane & 7) == 0)
                            *reinterpret_cast<uint32_t*>(sm + GRP_OFF + ring * GRP_BYTES + (4 * quarter + (lane >> 3)) * 4) = e_g | (((valid >> lane) & 0xffu) << 8);
                        tmem_wait_st();
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) {
                            mbar_arrive(bar(B_SCALES + ring));
                            mbar_arrive(bar(B_SREADY + b));
                            mbar_arrive_remote(barp(B_SCALEP + b));
                        }
                        ++sit;
                    }
                    there = idx >= 0;
                    if (there) sc = ld_in(reinterpret_cast<const uint4*>(p.kv + (size_t)idx * ROW_BYTES + SCALE_OFF));
                    idx = ahead.next_tile(p, meta) ? ahead.row_index(p, 32 * quarter + lane) : -1;
                    primed += filling ? 1u : 0u;
                }
                if (!ok) break;
                if (j == 0 && have && !scaler) {
                    // ---- q into shared memory
                    if (rq > 0) ok = mbar_wait_lean(bar(B_QFREE), (rq - 1) & 1u, abort_addr, WD_QFREE);   // the last one has been read for the last time
                    if (ok && rq > 0) ok = mbar_wait_lean(bar(B_QPART + quarter), (rq - 1) & 1u, abort_addr, WD_QPART);
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll 1
                    for (int i = 0; rq > 0 && i < 20; i += 4) {
                        uint32_t w[16];
                        tmem_ld16(lane_addr + TM_Q + 4 * i, w);
                        tmem_wait_ld();
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const uint32_t h = 16 * quarter + (i < 16 ? i + k : 4 * k + (lane >> 3));      // the last round: RoPE
                            *reinterpret_cast<uint4*>(sm + Q_OFF + (i < 16 ? lane >> 3 : 4) * CHUNK + swz(h, (uint32_t)lane & 7u)) =
                                make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
                        }
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(bar(B_QSCALE + (rq & (REQ_RING - 1))));
                        mbar_arrive_remote(barp(B_QREADYP));
                    }
                }
                if (j == j_epi && prev) {
                    // ---- epilogue of the request before
                    const uint32_t done = it - 1, pr = (rq - 1) & 1u;
                    ok = mbar_wait_lean(bar(B_SUMS + pr), ((rq - 1) >> 1) & 1u, abort_addr, WD_SUMS);
                    if (ok) ok = mbar_wait_lean(bar(B_PVDONE + (done & 1u)), (done >> 1) & 1u, abort_addr, WD_PVDONE);
                    if (!ok) break;
                    tc_fence_after();
                    const float* sums = reinterpret_cast<const float*>(sm + SUM_OFF + pr * SUM_BYTES);
                    const float l_all = (sums[hrow] + sums[64 + hrow]) + (sums[128 + hrow] + sums[192 + hrow]);
                    const float xm = fmaxf(fmaxf(sums[256 + hrow], sums[320 + hrow]), fmaxf(sums[384 + hrow], sums[448 + hrow])), m = sums[512 + hrow];
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar(B_SUMFREE + pr));
                    float lse = (l_all > 0.f) ? (log2f(l_all) - (float)P_SHIFT + m) : NEG_BIG;
                    float denom = l_all;
                    if (whole && p.attn_sink != nullptr && live) {
                        const float sink2 = p.attn_sink[head] * LOG2E;
                        denom = l_all + ((m == -INFINITY) ? INFINITY : exp2f(sink2 - m + (float)P_SHIFT));
                        if (lse != NEG_BIG) lse += log2f(1.f + exp2f(sink2 - lse));
                        else lse = sink2;
                    }
                    const float inv = (denom > 0.f) ? 1.f / denom : 0.f;
                    const size_t row = (size_t)(whole ? prev_req : meta.begin_split) * p.num_heads + (live ? head : 0);
                    // bf16 outputs, or fp16 records of equal partitions (the library's own scratch: a normalised partial is bounded by the
                    // largest |V|, and its rounding is an eighth of the output's); first output dim of this thread
                    uint8_t* dst = (whole ? reinterpret_cast<uint8_t*>(p.out) : reinterpret_cast<uint8_t*>(p.o_accum)) + (row * D_V + thalf * 256 + ch * 128) * 2;
                    const bool sectors = (reinterpret_cast<size_t>(dst) & 31) == 0;
                    auto accumulator_read = [&]() {        // the next request's first P.V may overwrite it
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_remote(barp(B_OFREEP));
                    };
#pragma unroll 1
                    for (int c = 0; c < 128; c += 32) {
                        uint32_t pk[16];
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            uint32_t o[16];
                            tmem_ld16(lane_addr + TM_O + 128 * ch + c + 16 * k, o);
                            tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                const float a = __uint_as_float(o[2 * i]) * inv, e = __uint_as_float(o[2 * i + 1]) * inv;
                                if (whole) {
                                    const __nv_bfloat162 t = __floats2bfloat162_rn(a, e);
                                    pk[8 * k + i] = *reinterpret_cast<const uint32_t*>(&t);
                                } else {
                                    const __half2 t = __floats2half2_rn(a, e);
                                    pk[8 * k + i] = *reinterpret_cast<const uint32_t*>(&t);
                                }
                            }
                        }
                        if (c == 96) accumulator_read();
                        if (!live) continue;
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const uint32_t v8[8] = {pk[8 * k], pk[8 * k + 1], pk[8 * k + 2], pk[8 * k + 3], pk[8 * k + 4], pk[8 * k + 5], pk[8 * k + 6], pk[8 * k + 7]};
                            if (sectors) {
                                st_global_v8(dst + 2 * c + 32 * k, v8);
                            } else {
                                *reinterpret_cast<uint4*>(dst + 2 * c + 32 * k) = make_uint4(v8[0], v8[1], v8[2], v8[3]);
                                *reinterpret_cast<uint4*>(dst + 2 * c + 32 * k + 16) = make_uint4(v8[4], v8[5], v8[6], v8[7]);
                            }
                        }
                    }
                    if (live && thalf == 0 && ch == 0) {
                        if (whole) {
                            p.out_lse[row] = lse;
                            if (p.out_max_logits) p.out_max_logits[row] = (xm == -INFINITY) ? NEG_BIG : xm;
                        } else {
                            p.lse_accum[row] = lse;
                        }
                    }
                }
            }
            if (!ok || !have) break;
            prev = true;
            prev_req = tiles.req;
            it += (uint32_t)tiles.nst;
            ++rq;
        }
        if (scaler && !together) named_bar_or(NB_SCALE, 128, !ok);     // (nobody stays behind at their barrier)
    } else if (warp == QK_WARP) {
        // =================================================================== score MMAs (odd CTA: its K rows have landed)
        Walk tiles(p, first, step, last);
        uint32_t it = 0, rq = 0;
        bool ok = true;
        const uint32_t q_lo = desc_lo(base + Q_OFF, 16);
        for (; ok && tiles.next_tile(p, meta); ++it) {
            const uint32_t b = it & 1u, ph = (it >> 1) & 1u;
            if (rank == 0) {
                if (tiles.j == 0) ok = mbar_wait_lean(bar(B_QREADYP), rq++ & 1u, abort_addr, WD_QREADY);
                // (the P.V of two tiles ago: with the scores the softmax warps also get the buffer of their weights)
                if (ok && it >= 2) ok = mbar_wait_lean(bar(B_SFREEP + b), ph ^ 1u, abort_addr, WD_SFREE);
                if (ok && it >= 2) ok = mbar_wait_lean(bar(B_PVDONE + b), ph ^ 1u, abort_addr, WD_PVDONE);
                if (ok) ok = mbar_wait_lean(bar(B_SCALEP + b), ph, abort_addr, WD_SCALES);
                if (ok) ok = mbar_wait_lean(bar(B_KPEERP + b), ph, abort_addr, WD_KPEER);
            }
            if (ok) ok = mbar_wait_lean(bar(B_KFULL + b), ph, abort_addr, WD_KFULL);
            if (!ok) break;
            if (rank != 0) {
                if (lane == 0) mbar_arrive_remote(barp(B_KPEERP + b));
                continue;
            }
            tc_fence_after();
            if (elect_one()) {
                const uint32_t k_lo = desc_lo(base + KS_OFF + b * KS_BYTES, 16), d = tmem + TM_S + 64 * b;
#pragma unroll 1
                for (int kc = 0; kc < 4; ++kc) {
                    const uint32_t a = q_lo + ((kc * CHUNK) >> 4), k = k_lo + ((kc * CHUNK) >> 4), idesc = idesc_mx(0) | ((uint32_t)kc << 4);
#pragma unroll
                    for (int s = 0; s < 4; ++s)
                        mma_pair_mxf8(d, make_desc(a + 2 * s, HI_128), make_desc(k + 2 * s, HI_128), idesc, tmem + TM_SFA, tmem + TM_SFB + 4 * b, (kc | s) != 0);
                }
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    mma_pair_f16(d, make_desc(q_lo + ((4 * CHUNK) >> 4) + 2 * s, HI_128), make_desc(k_lo + ((4 * CHUNK) >> 4) + 2 * s, HI_128), IDESC_ROPE, true);
                tc_commit_pair(bar(B_SREADY + b));
                tc_commit_pair(mapa_shared(bar(B_SREADY + b), 1));
                if (tiles.j + 1 == tiles.nst) {
                    tc_commit_pair(bar(B_QFREE));
                    tc_commit_pair(mapa_shared(bar(B_QFREE), 1));
                }
            }
            __syncwarp();
        }
    } else if (warp == PV_WARP) {
        if (rank == 0) {
            // ================================================================ P.V MMAs, half a tile at a time
            Walk tiles(p, first, step, last);
            uint32_t it = 0, rq = 0;
            bool ok = true;
            const uint32_t pb_lo = desc_lo(base + PB_OFF, 16), vs_lo = desc_lo(base + VS_OFF, V_STEP);
            for (; ok && tiles.next_tile(p, meta); ++it) {
                const uint32_t b = it & 1u;
                if (tiles.j == 0) {
                    if (rq > 0) ok = mbar_wait_lean(bar(B_OFREEP), (rq - 1) & 1u, abort_addr, WD_OFREE);
                    ++rq;
                }
                if (ok) ok = mbar_wait_lean(bar(B_PREADYP + b), (it >> 1) & 1u, abort_addr, WD_PREADY);
#pragma unroll 1
                for (uint32_t h = 0; ok && h < 2; ++h) {
                    const uint32_t slot = 2 * b + h;
                    ok = mbar_wait_lean(bar(B_VREADYP + slot), (it >> 1) & 1u, abort_addr, WD_VREADY);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t pa = pb_lo + ((b * CHUNK + h * 64) >> 4), va = vs_lo + ((slot * VS_BYTES) >> 4);
#pragma unroll
                        for (int kb = 0; kb < 2; ++kb) {
#pragma unroll
                            for (int nb = 0; nb < 2; ++nb)
                                mma_pair_f8(tmem + TM_O + 128 * nb, make_desc(pa + 2 * kb, HI_128), make_desc(va + ((nb * V_BLOCK + kb * V_STEP) >> 4), HI_128),
                                            IDESC_PV, ((uint32_t)tiles.j | h | (uint32_t)kb) != 0u);
                        }
                        tc_commit_pair(bar(B_VFREE + slot));
                        tc_commit_pair(mapa_shared(bar(B_VFREE + slot), 1));
                        if (h == 1) {
                            tc_commit_pair(bar(B_PVDONE + b));
                            tc_commit_pair(mapa_shared(bar(B_PVDONE + b), 1));
                        }
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp >= FIX_WARP0) {
        // =================================================================== V onto the groups' scales
        // Each warp looks after 16 rows x two blocks of 128 dims of every tile, a lane after one of these pieces.  Those that have another
        // scale than their group are listed first, then eight lanes take one each: the ALU pipe, which takes an instruction
        // every other cycle, is what this costs.
        const uint32_t f = warp - FIX_WARP0, h = f >> 2, at0 = (lane >> 4) * V_BLOCK + (16 * (f & 3u) + (lane & 15)) * 128;
        uint32_t* list = reinterpret_cast<uint32_t*>(sm + FIX_OFF) + f * FIX_LIST;
        for (uint32_t i = lane; i < FIX_LIST; i += 32) list[i] = 0u;      // (entries past the end are read, not written back)
        __syncwarp();
        Walk tiles(p, first, step, last);
        bool ok = true;
        for (uint32_t it = 0; tiles.next_tile(p, meta); ++it) {
            const uint32_t ring = it & (REC_RING - 1), slot = 2 * (it & 1u) + h;
            ok = mbar_wait_lean(bar(B_SCALES + ring), (it / REC_RING) & 1u, abort_addr, WD_SCALES);
            const uint32_t rec = (uint32_t)reinterpret_cast<const uint16_t*>(sm + REC_OFF)[ring * TILE_N + 16 * f + (lane & 15)];
            // the pieces of 128 bytes (a token's block) to be shifted: where | by how much << 14
            const uint32_t d = (rec >> (8 * rank + 4 * (lane >> 4))) & 15u, todo = __ballot_sync(0xffffffffu, d != 0u);
            const int n = __popc(todo);
            if (d != 0u) list[__popc(todo & ((1u << lane) - 1u))] = at0 | (d << 14);
            __syncwarp();
            if (ok) ok = mbar_wait_lean(bar(B_VFULL + slot), (it >> 1) & 1u, abort_addr, WD_VFULL);
            if (!ok) break;
            uint8_t* v0 = sm + VS_OFF + slot * VS_BYTES + (lane & 7) * 16;
#pragma unroll 1
            for (int i = 0; i < n; i += 16) {
                uint4 v[4];
                uint8_t* at[4];
                uint32_t sub[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint32_t e = list[i + 4 * u + (lane >> 3)];
                    at[u] = v0 + (e & 0x3fffu);
                    sub[u] = (e >> 14) * 0x08080808u;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = *reinterpret_cast<const uint4*>(at[u]);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    v[u].x = shift_down_e4m3x4(v[u].x, sub[u]); v[u].y = shift_down_e4m3x4(v[u].y, sub[u]);
                    v[u].z = shift_down_e4m3x4(v[u].z, sub[u]); v[u].w = shift_down_e4m3x4(v[u].w, sub[u]);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (i + 4 * u + (lane >> 3) < n) *reinterpret_cast<uint4*>(at[u]) = v[u];
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(barp(B_VREADYP + slot));
        }
    } else {
        // =================================================================== rows -> K stages, V slots
        // Two warps gather this CTA's 64 rows whole (four blocks and the RoPE) for K, four all rows' dims [256 rank, +256) for V, 32 rows
        // each.  The lanes read the rows' numbers ahead and hand them to the lane that issues the copies through shared memory:
        // passed by shuffles, under an election for every four rows, they made the copies a third of all instructions.
        const bool is_k = warp < V_WARP0;
        const uint32_t w = is_k ? warp - COPY_WARP0 : warp < QK_WARP ? warp - V_WARP0 : warp - PV_WARP + 1;      // K: 0, 1; V: 0 to 3
        const int row0 = (is_k ? OWN_N * (int)rank : 0) + 32 * (int)w + lane;
        int* mine = reinterpret_cast<int*>(sm + IDX_OFF) + 32 * (is_k ? w : 2 + w);
        Walk tiles(p, first, step, last);
        bool ok = true;
        int idx = 0;
        uint32_t it = 0;
        for (bool have = true, warm = false; have; warm = true) {
            mine[lane] = idx >= 0 ? idx : NO_ROW;
            have = tiles.next_tile(p, meta);
            idx = have ? tiles.row_index(p, row0) : -1;    // read ahead of its use
            if (!warm) continue;
            const uint32_t b = it & 1u, slot = 2 * b + (w >> 1);
            if (it >= 2) ok = mbar_wait_lean(is_k ? bar(B_SREADY + b) : bar(B_VFREE + slot), ((it >> 1) - 1) & 1u, abort_addr, is_k ? WD_SREADY : WD_VFREE);
            if (!ok) break;
            __syncwarp();
            if (elect_one()) {
                if (is_k) {
                    uint32_t dst = base + KS_OFF + b * KS_BYTES + w * (32 * 128);
                    const uint32_t full = bar(B_KFULL + b);
                    mbar_arrive_expect_tx(full, 5 * 32 * 128);
#pragma unroll 1
                    for (int q = 0; q < 32; q += 4, dst += 512) {
                        const int4 i = *reinterpret_cast<const int4*>(mine + q);
#pragma unroll
                        for (uint32_t c = 0; c < 5; ++c) tma_gather4(dst + c * CHUNK, &kv_map, (int)(c < 4 ? 32 * c : ROPE_OFF / 4), i.x, i.y, i.z, i.w, full);
                    }
                } else {
                    uint32_t dst = base + VS_OFF + slot * VS_BYTES + (w & 1u) * (32 * 128);
                    const uint32_t full = bar(B_VFULL + slot);
                    mbar_arrive_expect_tx(full, 2 * 32 * 128);
#pragma unroll 1
                    for (int q = 0; q < 32; q += 4, dst += 512) {
                        const int4 i = *reinterpret_cast<const int4*>(mine + q);
#pragma unroll
                        for (uint32_t c = 0; c < 2; ++c) tma_gather4(dst + c * V_BLOCK, &kv_map, (int)(64 * rank + 32 * c), i.x, i.y, i.z, i.w, full);
                    }
                }
            }
            __syncwarp();
            ++it;
        }
    }

    // ------------------------------------------------------------------------ teardown
    if (*abort_flag != 0) {        // a wait gave up: copies and MMAs may still be in flight; give them time to finish
        const long long t0 = clock64();
        while (clock64() - t0 < 200000) { }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();        // the partner may still arrive on this CTA's barriers until here
    if (tid == 0 && *abort_flag != 0 && p.status != nullptr) {
        atomicCAS(p.status, 0, *abort_flag);
        atomicAdd(p.status + 1, 1);
        p.status[2] = blockIdx.x;
    }
    if (warp == QK_WARP) {
        tc_fence_after();
        tmem_dealloc_pair(tmem, TMEM_COLS);
    }
}

}  // namespace

// 65 to 128 heads (and the longer lists of fewer heads that attn_tile_kernel leaves) over one linear array of rows, where this kernel is
// the faster one.  us here / in the pair kernel, 128 heads, rows in HBM:
//   whole requests        64 of 2048 entries 47.0 / 49.4, 16: 39.3 / 44.2; 48 of 1024: 29.0 / 29.0, 16: 25.7 / 29.0; 16 of 512: 18.9 / 20.8
//   several per pair      4096 of 2048 entries 1920 / 2240, 740: 305 / 398, 740 of 1024: 228 / 241; but 740 of 768 217 / 200, of 512 171 / 163,
//                         of 128 126 / 124: the q of the next request takes this kernel longer, which short lists do not hide.  With one
//                         to four short requests per pair there is less of that: 148 of 512 33 / 38, of 64 22 / 30.
//   equal partitions      1 request of 2048 in 8: 22.8 / 22.9, 4 in 8: 22.8 / 24.8, 16 in 4: 27.8 / 28.9, 32 in 2: 35.1 / 35.1
//   scheduler's           13 ragged requests of 2048 in 52: 33.4 / 31.0, 20 in 74: 37.6 / 35.1 (24 in 74 43.4 / 46.3, but whole they take
//                         39.0): partitions that straddle two requests are short lists.
bool attn_duo_takes(const AttnParams& p) {
    if (p.num_heads > 128 || p.sched != nullptr || !one_linear_array(p) || attn_tile_takes(p)) return false;
    return p.uniform_k > 1 || p.topk > 15 * BLOCK_N || p.num_tokens <= 4 * (smla_num_sms() / 2);
}

int launch_attn_duo(const AttnParams& p, cudaStream_t stream) {
    if (p.num_tokens == 0) return 0;
    static std::atomic<bool> attr_set[64];
    static int sm_count[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return set_error(SMLA_E_SHAPE, "attn_duo_kernel: device ordinal %d not supported", dev);
    if (!attr_set[dev]) {
        cudaFuncAttributes fa;
        if (cudaFuncGetAttributes(&fa, attn_duo_kernel) != cudaSuccess || fa.numRegs != REGS_LAUNCH)
            return set_error(SMLA_E_DEVICE, "attn_duo_kernel: compiled with %d registers per thread, the warpgroup budgets assume %d",
                             fa.numRegs, REGS_LAUNCH);
        const cudaError_t e = cudaFuncSetAttribute(attn_duo_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_ALLOC);
        if (e != cudaSuccess) return set_error((int)e, "attn_duo_kernel: cannot reserve %u bytes of shared memory: %s", SMEM_ALLOC, cudaGetErrorString(e));
        cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev);
        attr_set[dev] = true;
    }
    CUtensorMap map;
    if (int e = rows_tensor_map(p.kv, &map)) return e;
    const int max_pairs = sm_count[dev] >= 2 ? sm_count[dev] / 2 : 1;
    const int parts = p.uniform_k > 1 ? p.uniform_k * p.num_tokens : (p.num_tokens < max_pairs ? p.num_tokens : max_pairs);
    launch_dependent(attn_duo_kernel, dim3(2 * parts), dim3(DUO_THREADS), SMEM_ALLOC, stream, p, map);
    return check_launch("attn_duo_kernel");
}

}  // namespace smla

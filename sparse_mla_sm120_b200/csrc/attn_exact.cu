// Exact sparse-MLA attention over the MODEL1 cache layout on tcgen05 (sm_100a): decode with split-KV and prefill, one or
// two caches.  Nothing is rounded below bf16 inputs and fp32 sums:
//   * a cache row is dequantised to the bf16 values the layout stands for (e4m3 x power of two and bf16 RoPE: exact),
//     q is bf16 as given: the products of the score MMAs are exact and summed in fp32;
//   * softmax in fp32; a weight enters P.V as the sum of two bf16 numbers (hi + lo, off by at most 2^-17 of the weight),
//     each multiplied exactly and summed in fp32; the denominator sums the fp32 weights.
//
// Work unit: one scheduler partition (a run of 64-token blocks of consecutive requests, see sched.cu; without a scheduler:
// a contiguous share of the requests) for 64 query heads; up to 128 heads are two CTAs.  Both contractions run
// transposed, so that every MMA has M = 128 whatever the number of heads, and the gathered rows are the A operand of
// both without being moved or copied:
//   * S^T [128 tokens x 64 heads] = K [tokens x 512 dims] . Q^T: A = the tile of rows, K-major, B = Q;
//   * O^T [4 x 128 dims x 64 heads] += V^T . P: A = the same tile read MN-major (V is the whole row in this layout),
//     B = the weights, one 128-byte line of 64 heads per token, hi and lo one after the other.
// Tensor memory: O^T 256 columns, S^T 64.  Shared memory: rows 128 KB (bf16, eight chunks of 64 dims, 128B swizzle),
// Q 64 KB, weights 2 x 16 KB.
//
// Warp roles (896 threads):
//   warps 0-7    softmax, epilogue and Q: warp w holds tokens [32 (w % 4), +32) and heads [32 (w / 4), +32) of a tile, a
//                thread one token; maxima over tokens by redux across the lanes, lane i keeps the state of head i.
//   warps 8-23   gather: warp g dequantises eight rows of every tile, two of each quarter of 32 tokens.  The next tile's rows are loaded into registers
//                while the MMAs work on this one.
//   warp 24      issues the MMAs (one elected lane).
// What bounds it: the phases of a tile (rows -> scores -> softmax -> P.V) follow each other, about 11000 cycles per 128
// tokens, since the rows as bf16 leave no room for a second tile.  Shared memory is the resource: 96 MMAs at N = 64 read
// 6 KB each (49 cycles, measured), the rows are another 128 KB written.  The conversion of the next tile therefore starts
// as soon as P.V has read a quarter of this one, and its loads (which registers and L1 hold only in part) are sent ahead by
// an L2 prefetch two tiles away.  32 requests of 128 heads, up to 1024 entries and a second cache of 128: 51 us; the
// CUDA-core kernel that served this layout before took 1924 us.
// Every wait is bounded; a wait that gives up records a code in status[] and the CTA drains and exits.
#include "attn_common.cuh"
#include "sm100_ptx.cuh"

namespace smla {

namespace {

using namespace ptx;
using namespace attn;

constexpr int X_DIM = SMLA_M1_D_QK;             // 512 dims of q, K and V
constexpr int X_NOPE = 448, X_DATA = SMLA_M1_DATA_BYTES;
constexpr int X_HEADS = 64;                     // heads per CTA
constexpr int X_TILE = 128;                     // tokens per tile: two scheduler blocks
constexpr int X_SM_WARPS = 8, X_G_WARPS = 16, X_RPW = X_TILE / X_G_WARPS;
constexpr int X_MMA_WARP = X_SM_WARPS + X_G_WARPS;
constexpr int X_THREADS = (X_MMA_WARP + 4) * 32;
constexpr int X_REGS_LAUNCH = 72, X_REGS_SOFTMAX = 112, X_REGS_GATHER = 64, X_REGS_MMA = 24;
static_assert(X_SM_WARPS * 32 * X_REGS_SOFTMAX + X_G_WARPS * 32 * X_REGS_GATHER + 128 * X_REGS_MMA <= X_THREADS * X_REGS_LAUNCH,
              "register budgets exceed what the CTA owns");
static_assert(65536 / X_THREADS / 8 * 8 == X_REGS_LAUNCH, "launch-time registers per thread");
// The running maximum of a head lags by at most 2^X_TAU: sums and weights are floating point, so a lagging maximum costs
// no precision, and the accumulator is rescaled only a few times per request.
constexpr float X_TAU = 16.0f;

constexpr uint32_t XK_CHUNK = X_TILE * 128;                   // 64 dims of all rows
constexpr uint32_t XQ_CHUNK = X_HEADS * 128;                  // 64 dims of all heads
constexpr uint32_t XK_OFF = 0;
constexpr uint32_t XQ_OFF = XK_OFF + 8 * XK_CHUNK;
constexpr uint32_t XP_OFF = XQ_OFF + 8 * XQ_CHUNK;            // hi, then lo: [128 tokens x 64 heads] bf16
constexpr uint32_t XP_BYTES = X_TILE * 128;
constexpr uint32_t XV_OFF = XP_OFF + 2 * XP_BYTES;            // validity: one bit per token, [2 tiles][16 gather warps] bytes
constexpr uint32_t XX_OFF = XV_OFF + 2 * X_G_WARPS;           // exchange between the softmax warps of 32 heads: [4][64] fp32
constexpr uint32_t XM_OFF = XX_OFF + 4 * X_HEADS * 4;         // running maxima [64] fp32 (the four warps of a head write the same value)
constexpr uint32_t XB_OFF = XM_OFF + X_HEADS * 4;
constexpr int XB_KFULL = 0, XB_SREADY = 1, XB_PREADY = 2, XB_PVDONE = 3, XB_QREADY = 4,
              XB_KFREE = 5, XB_N = 9;                                 // KFREE: P.V has read the tile's tokens [32 i, +32)
constexpr uint32_t XMISC_OFF = XB_OFF + XB_N * 8;
constexpr uint32_t X_SMEM = XMISC_OFF + 16 + 1024;
static_assert(X_SMEM <= 227 * 1024, "shared memory budget");
static_assert(XB_OFF % 8 == 0 && XX_OFF % 16 == 0 && XM_OFF % 16 == 0, "alignment");

constexpr uint32_t XT_O = 0, XT_S = 256;                      // tensor memory: dims block b of O^T at 64 b, scores at 256
constexpr uint32_t IDESC_S = instr_desc(FMT_BF16, FMT_BF16, false, false, 128, X_HEADS);
constexpr uint32_t IDESC_O = instr_desc(FMT_BF16, FMT_BF16, true, true, 128, X_HEADS);
constexpr uint32_t X_DESC_HI = desc_hi(1024, (uint32_t)SWIZZLE_128B);

enum { WX_KFREE = 41, WX_KFULL = 42, WX_SREADY = 43, WX_PREADY = 44, WX_PVDONE = 45, WX_QREADY = 46 };

__device__ __forceinline__ uint32_t xswz(uint32_t row, uint32_t piece) { return row * 128u + ((piece ^ (row & 7u)) << 4); }

// Largest value over the lanes of the warp (redux on fp32; -inf where no lane has a larger one).
__device__ __forceinline__ float redux_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// Four e4m3 values times 2^-120 as two bf16 pairs, (v0, v2) and (v1, v3): the same bits in other places (subnormals
// included).  Pairing every other value saves the byte permutations; the integer pipe is what the conversion is bound by.
// So the dims of a row lie in shared memory with the middle two of every four exchanged (RoPE excepted), q is stored the
// same way and the epilogue undoes it.
__device__ __forceinline__ void e4m3_as_bf16(uint32_t w, uint32_t& even, uint32_t& odd) {
    even = ((w * 256u) & 0x80008000u) | ((w * 16u) & 0x07f007f0u);
    odd = (w & 0x80008000u) | ((w >> 4) & 0x07f007f0u);
}
// Bit 7 of every byte: whether the e4m3 value is no number (all seven lower bits set).
__device__ __forceinline__ uint32_t no_number_bytes(uint32_t w) { return (w & 0x7f7f7f7fu) + 0x01010101u; }
__device__ __forceinline__ int exact_dim_at(int pos) {           // output dim of position pos of a row, and the reverse
    return (pos < X_NOPE && ((pos + 1) & 2)) ? pos ^ 3 : pos;
}
// 2^n as a pair of bf16 numbers, -126 <= n <= 127.
__device__ __forceinline__ __nv_bfloat162 pow2_bf16x2(uint32_t n_biased) {
    const uint32_t b = (n_biased << 7) * 0x00010001u;
    return *reinterpret_cast<const __nv_bfloat162*>(&b);
}

// The CTA's share of the work: a scheduler record, or a contiguous run of whole requests.
__device__ __forceinline__ SchedMeta exact_meta(const AttnParams& p) {
    if (p.sched != nullptr) return p.sched[blockIdx.x];
    SchedMeta m;
    m.begin_req = (int)((long long)blockIdx.x * p.num_tokens / gridDim.x);
    m.end_req = (int)((long long)(blockIdx.x + 1) * p.num_tokens / gridDim.x) - 1;
    m.begin_block = 0; m.end_block = 0x7fffffff;
    m.begin_split = 0; m.first_split = m.last_split = 0; m.pad = 0;
    return m;
}

// The tiles of the CTA's requests, one after the other.
struct TileWalk {
    Work w;
    int req, j, nst;
    __device__ __forceinline__ explicit TileWalk(int begin_req) : req(begin_req - 1), j(0), nst(0) {}
    __device__ __forceinline__ bool next(const AttnParams& p, const SchedMeta& meta, int last_req) {
        if (++j < nst) return true;
        j = nst = 0;
        do { if (++req > last_req) { req = last_req; return false; } } while (!get_work(p, meta, req, w));
        nst = (w.nblk + 1) >> 1;
        return true;
    }
};

__global__ void __launch_bounds__(X_THREADS, 1) attn_exact_kernel(const AttnParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* sm = smem_raw + (base - raw);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + XMISC_OFF + 4);
    const uint32_t abort_addr = base + XMISC_OFF + 4;
    auto bar = [&](int i) -> uint32_t { return base + XB_OFF + 8u * i; };
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int head0 = (int)blockIdx.y * X_HEADS;

    if (tid == 0) {
        mbar_init(bar(XB_KFULL), X_G_WARPS);
        mbar_init(bar(XB_SREADY), 1);
        mbar_init(bar(XB_PREADY), X_SM_WARPS);
        mbar_init(bar(XB_PVDONE), 1);
        mbar_init(bar(XB_QREADY), X_SM_WARPS);
        for (int i = 0; i < 4; ++i) mbar_init(bar(XB_KFREE + i), 1);
        *abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == X_MMA_WARP) { tmem_alloc(base + XMISC_OFF, 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(sm + XMISC_OFF);
    grid_dep_wait();
    grid_dep_launch();
    const SchedMeta meta = exact_meta(p);
    const int last_req = min(meta.end_req, p.num_tokens - 1);
    if (warp < X_SM_WARPS) setmaxnreg_inc<X_REGS_SOFTMAX>();
    else if (warp < X_MMA_WARP) setmaxnreg_dec<X_REGS_GATHER>();
    else setmaxnreg_dec<X_REGS_MMA>();

    if (warp < X_SM_WARPS) {
        // =================================================================== softmax + epilogue + Q
        const int quarter = warp & 3, half = warp >> 2;
        const int token = quarter * 32 + lane;             // of the tile; in O^T: output dim inside a block of 128
        const int hl = half * 32 + lane;                   // the head whose state this lane keeps (the same in four warps)
        const bool live = head0 + hl < p.num_heads;
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
        float* xx = reinterpret_cast<float*>(sm + XX_OFF);
        float* xm = reinterpret_cast<float*>(sm + XM_OFF);
        const float c = p.sm_scale * LOG2E;
        uint32_t it = 0;
        bool dead = false, stop = false;
        for (int req = meta.begin_req; req <= last_req && !stop; ++req) {
            Work w;
            if (!get_work(p, meta, req, w)) continue;
            const int nst = (w.nblk + 1) >> 1;
            // ---- Q: [64 heads x 512 dims], K-major, eight chunks of 64 dims; the previous request's last score MMAs are done
            {
                const __nv_bfloat16* q0 = p.q + ((size_t)req * p.num_heads + head0) * X_DIM;
#pragma unroll 1
                for (int u = 0; u < 16; u += 8) {
                    uint4 v[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int i = tid + (u + k) * (X_SM_WARPS * 32), h = i >> 6;
                        v[k] = make_uint4(0, 0, 0, 0);
                        if (head0 + h < p.num_heads) v[k] = ld_in(reinterpret_cast<const uint4*>(q0 + (size_t)h * X_DIM + (i & 63) * 8));
                    }
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int i = tid + (u + k) * (X_SM_WARPS * 32), h = i >> 6, pc = i & 63;
                        if (pc < X_NOPE / 8)                // the order of e4m3_as_bf16
                            v[k] = make_uint4(__byte_perm(v[k].x, v[k].y, 0x5410), __byte_perm(v[k].x, v[k].y, 0x7632),
                                              __byte_perm(v[k].z, v[k].w, 0x5410), __byte_perm(v[k].z, v[k].w, 0x7632));
                        *reinterpret_cast<uint4*>(sm + XQ_OFF + (pc >> 3) * XQ_CHUNK + xswz((uint32_t)h, (uint32_t)pc & 7u)) = v[k];
                    }
                }
                fence_proxy_async();
            }
            float m_run = -INFINITY, x_max = -INFINITY;     // of head hl
            float l[32];                                    // this token's share of the denominators of the warp's 32 heads
#pragma unroll
            for (int i = 0; i < 32; ++i) l[i] = 0.f;
            xm[hl] = 0.f;
            tc_fence_before();                              // the previous epilogue's reads of the accumulator
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(XB_QREADY));
            for (int j = 0; j < nst; ++j, ++it) {
                uint32_t sv[32];
                bool valid = false;
                if (!dead) dead = !mbar_wait_lean(bar(XB_SREADY), it & 1u, abort_addr, WX_SREADY);
                if (!dead) {
                    tc_fence_after();
                    tmem_ld32(lane_addr + XT_S + 32 * half, sv);
                    valid = (sm[XV_OFF + (it & 1u) * X_G_WARPS + ((token & 31) >> 1)] >> (2 * quarter + (token & 1))) & 1;
                    tmem_wait_ld();
                    float mine = -INFINITY;
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const float r = redux_max(valid ? __uint_as_float(sv[i]) * c : -INFINITY);
                        if (lane == i) mine = r;
                    }
                    xx[quarter * X_HEADS + hl] = mine;
                }
                if (named_bar_or(1 + half, 128, dead || *abort_flag != 0)) { stop = true; break; }
                const float mx = fmaxf(fmaxf(xx[hl], xx[X_HEADS + hl]), fmaxf(xx[2 * X_HEADS + hl], xx[3 * X_HEADS + hl]));
                x_max = fmaxf(x_max, mx);
                const bool grow = mx > m_run + X_TAU;       // false while the head has seen no entry
                if (__any_sync(0xffffffffu, grow)) {
                    const float alpha = grow ? ex2(m_run - mx) : 1.f;     // 0 for the first entries
                    if (grow) m_run = mx;
                    xm[hl] = m_run == -INFINITY ? 0.f : m_run;
#pragma unroll
                    for (int i = 0; i < 32; ++i) l[i] *= __shfl_sync(0xffffffffu, alpha, i);
                    if (j > 0) {                            // scores of this tile are ready: P.V of the last one has completed
#pragma unroll 1
                        for (int b = 0; b < 4; ++b) {
                            uint32_t o[32];
                            tmem_ld32(lane_addr + XT_O + 64 * b + 32 * half, o);
                            tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * __shfl_sync(0xffffffffu, alpha, i));
                            tmem_st32(lane_addr + XT_O + 64 * b + 32 * half, o);
                        }
                        tmem_wait_st();
                    }
                }
                __syncwarp();
#pragma unroll
                for (int k = 0; k < 4; ++k) {               // eight heads: one 16-byte piece of the token's lines
                    uint32_t hi[4], lo[4];
#pragma unroll
                    for (int e = 0; e < 4; e += 2) {
                        const float4 m4 = *reinterpret_cast<const float4*>(xm + half * 32 + 8 * k + 2 * e);
                        const float mm[4] = {m4.x, m4.y, m4.z, m4.w};
                        float pv[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int h = 8 * k + 2 * e + i;
                            pv[i] = valid ? ex2(fmaf(__uint_as_float(sv[h]), c, -mm[i])) : 0.f;
                            l[h] += pv[i];
                        }
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const __nv_bfloat162 a = __floats2bfloat162_rn(pv[2 * i], pv[2 * i + 1]);
                            const uint32_t au = *reinterpret_cast<const uint32_t*>(&a);
                            const __nv_bfloat162 r = __floats2bfloat162_rn(pv[2 * i] - bf16lo(au), pv[2 * i + 1] - bf16hi(au));
                            hi[e + i] = au;
                            lo[e + i] = *reinterpret_cast<const uint32_t*>(&r);
                        }
                    }
                    const uint32_t at = XP_OFF + xswz((uint32_t)token, (uint32_t)(half * 4 + k));
                    *reinterpret_cast<uint4*>(sm + at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                    *reinterpret_cast<uint4*>(sm + at + XP_BYTES) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                }
                fence_proxy_async();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(XB_PREADY));
            }
            if (stop) break;
            // ---- epilogue
            if (!dead) dead = !mbar_wait_lean(bar(XB_PVDONE), (it - 1) & 1u, abort_addr, WX_PVDONE);
            tc_fence_after();
            // sum over the warp's tokens: halve the list at every exchange, lane i ends with head i
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) {
#pragma unroll
                for (int i = 0; i < o; ++i) {
                    const bool up = (lane & o) != 0;
                    const float send = up ? l[i] : l[i + o], keep = up ? l[i + o] : l[i];
                    l[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
            xx[quarter * X_HEADS + hl] = l[0];
            if (named_bar_or(1 + half, 128, dead || *abort_flag != 0)) { stop = true; break; }
            const float l_all = (xx[hl] + xx[X_HEADS + hl]) + (xx[2 * X_HEADS + hl] + xx[3 * X_HEADS + hl]);
            float lse = (l_all > 0.f) ? (log2f(l_all) + m_run) : NEG_BIG;
            float denom = l_all;
            if (w.no_split && p.attn_sink != nullptr && live) {
                const float sink2 = p.attn_sink[head0 + hl] * LOG2E;
                denom = l_all + ((m_run == -INFINITY) ? INFINITY : exp2f(sink2 - m_run));
                if (lse != NEG_BIG) lse += log2f(1.f + exp2f(sink2 - lse));
                else lse = sink2;
            }
            const float inv = (denom > 0.f) ? 1.f / denom : 0.f;
            const size_t row0 = (size_t)(w.no_split ? req : w.split_idx) * p.num_heads + head0 + half * 32;
            const int n_live = min(p.num_heads - head0 - half * 32, 32);      // of the warp's heads
#pragma unroll 1
            for (int b = 0; b < 4; ++b) {
                uint32_t o[32];
                tmem_ld32(lane_addr + XT_O + 64 * b + 32 * half, o);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * __shfl_sync(0xffffffffu, inv, i));
                const int d = exact_dim_at(128 * b + token);
                // a head's 32 dims of the warp are one store of 64 (bf16) or 128 bytes
                auto store = [&](auto* dst, auto cvt) {
                    if (n_live == 32) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) dst[i * D_V] = cvt(__uint_as_float(o[i]));
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (i < n_live) dst[i * D_V] = cvt(__uint_as_float(o[i]));
                    }
                };
                if (w.no_split) store(p.out + row0 * D_V + d, [](float v) { return __float2bfloat16(v); });
                else store(p.o_accum + row0 * D_V + d, [](float v) { return v; });
            }
            if (live && quarter == 0) {
                if (w.no_split) {
                    p.out_lse[row0 + lane] = lse;
                    if (p.out_max_logits) p.out_max_logits[row0 + lane] = (x_max == -INFINITY) ? NEG_BIG : x_max;
                } else {
                    p.lse_accum[row0 + lane] = lse;
                }
            }
        }
    } else if (warp < X_MMA_WARP) {
        // =================================================================== gather
        const int g = warp - X_SM_WARPS;
        // Row i of the warp is a token of quarter i / 2 of the tile, so that all warps work on a quarter as soon as P.V has read it.
        auto token_of = [&](int i) -> int { return (i >> 1) * 32 + 2 * g + (i & 1); };
        TileWalk walk(meta.begin_req);
        uint4 nope[X_RPW], rp[X_RPW / 4];
        uint2 sc8 = make_uint2(0u, 0u);
        uint32_t vbits = 0u;
        auto load_rows = [&](int idx, bool extra) {         // idx: lane i holds the index of row i % 8
            uint32_t lo = 0u, hi = 0u;
            sc8 = make_uint2(0u, 0u);
            if (idx >= 0) {
                const uint8_t* kv = extra ? p.extra_kv : p.kv;
                const unsigned pbs = (unsigned)(extra ? p.extra_page_block_size : p.page_block_size);
                const unsigned blk = (unsigned)idx / pbs, in = (unsigned)idx - blk * pbs;
                const uint8_t* page = kv + (int64_t)blk * (extra ? p.extra_block_stride : p.block_stride);
                sc8 = ld_in(reinterpret_cast<const uint2*>(page + (int64_t)pbs * X_DATA + (int64_t)in * 8));
                const unsigned long long at = reinterpret_cast<unsigned long long>(page + (int64_t)in * X_DATA);
                lo = (uint32_t)at; hi = (uint32_t)(at >> 32);
            }
            vbits = __ballot_sync(0xffffffffu, idx >= 0) & ((1u << X_RPW) - 1u);
            auto row_at = [&](int r) -> const uint8_t* {
                const uint32_t a = __shfl_sync(0xffffffffu, lo, r), b = __shfl_sync(0xffffffffu, hi, r);
                return reinterpret_cast<const uint8_t*>(((unsigned long long)b << 32) | a);
            };
#pragma unroll
            for (int i = 0; i < X_RPW; ++i) {
                const uint8_t* row = row_at(i);
                nope[i] = make_uint4(0, 0, 0, 0);
                if (((vbits >> i) & 1u) && lane < X_NOPE / 16) nope[i] = ld_row16(row + lane * 16);
            }
#pragma unroll
            for (int u = 0; u < X_RPW / 4; ++u) {
                const int r = (lane >> 3) + 4 * u;
                const uint8_t* row = row_at(r);
                rp[u] = make_uint4(0, 0, 0, 0);
                if ((vbits >> r) & 1u) rp[u] = ld_row16(row + X_NOPE + (lane & 7) * 16);
            }
        };
        // Ask L2 for the rows of a tile that is two tiles away: registers and L1 hold only a part of a tile's rows in flight,
        // so those loads should find their rows in L2.
        auto prefetch_rows = [&](int idx, bool extra) {
            uint32_t lo = 0u, hi = 0u;
            if (idx >= 0) {
                const uint8_t* kv = extra ? p.extra_kv : p.kv;
                const unsigned pbs = (unsigned)(extra ? p.extra_page_block_size : p.page_block_size);
                const unsigned blk = (unsigned)idx / pbs, in = (unsigned)idx - blk * pbs;
                const uint8_t* page = kv + (int64_t)blk * (extra ? p.extra_block_stride : p.block_stride);
                const unsigned long long at = reinterpret_cast<unsigned long long>(page + (int64_t)in * X_DATA);
                lo = (uint32_t)at; hi = (uint32_t)(at >> 32);
                if (lane < X_RPW) asm volatile("prefetch.global.L2 [%0];" ::"l"(page + (int64_t)pbs * X_DATA + (int64_t)in * 8));
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {                   // row lane / 8 (+ 4 u), 128 bytes per lane
                const int r = (lane >> 3) + 4 * u;
                const uint32_t a = __shfl_sync(0xffffffffu, lo, r), b = __shfl_sync(0xffffffffu, hi, r);
                const unsigned off = min((unsigned)(lane & 7) * 128u, (unsigned)X_DATA - 1u);
                if ((a | b) != 0u && (lane & 7) < 6)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"((((unsigned long long)b << 32) | a) + off));
            }
        };
        bool extra = false;
        auto fetch = [&](bool have) -> int {
            if (!have) return -1;
            const int r = token_of(lane & (X_RPW - 1)), b = walk.w.blk0 + 2 * walk.j + (r >> 6);
            extra = b >= walk.w.main_blocks;                // of this lane's row
            return fetch_entry(p, walk.w, b, r & 63);
        };
        bool have = walk.next(p, meta, last_req), ok = true;
        int idx = fetch(have);
        bool extra_now = extra, have_next = false;
        load_rows(idx, extra_now);
        have_next = have && walk.next(p, meta, last_req);
        idx = fetch(have_next);                             // of the tile after this one
        extra_now = extra;
        prefetch_rows(idx, extra_now);
        const int bk = lane >> 2;                           // 64-value block, and chunk, of this lane's piece
        const bool odd = (lane & 4) != 0;
        for (uint32_t it = 0; have; ++it) {
            const bool have_after = have_next && walk.next(p, meta, last_req);
            int idx_after = fetch(have_after);              // read while this tile is stored
            // A byte that is no number (the conversion would make 480 of it) makes its token's score none: one pair of the row's
            // RoPE values, which every score and every weight's product meets, becomes NaN.  Looked for here, while P.V still
            // reads the tile before; in the conversion it cost 2 us of 51.
            uint32_t bad = 0u;
#pragma unroll
            for (int i = 0; i < X_RPW; ++i) {
                const uint32_t none = no_number_bytes(nope[i].x) | no_number_bytes(nope[i].y) | no_number_bytes(nope[i].z) | no_number_bytes(nope[i].w);
                bad |= __any_sync(0xffffffffu, (none & 0x80808080u) != 0u) ? 1u << i : 0u;
            }
            if (bad != 0u) {
#pragma unroll
                for (int u = 0; u < X_RPW / 4; ++u)
                    if ((bad >> ((lane >> 3) + 4 * u)) & 1u) rp[u].x = 0x7fff7fffu;
            }
#pragma unroll
            for (int i = 0; i < X_RPW; ++i) {
                if (it >= 1 && (i & 1) == 0 && ok) ok = mbar_wait_lean(bar(XB_KFREE + (i >> 1)), (it - 1) & 1u, abort_addr, WX_KFREE);
                const uint32_t w0 = __shfl_sync(0xffffffffu, sc8.x, i), w1 = __shfl_sync(0xffffffffu, sc8.y, i);
                const uint32_t e = (((bk & 4) ? w1 : w0) >> (8 * (bk & 3))) & 0xffu;
                // the block's scale 2^(e - 127) times the 2^120 of e4m3_as_bf16x2; what does not fit a bf16 power is made up below
                const __nv_bfloat162 f = pow2_bf16x2(min(e, 134u) + 120u);
                // neighbouring chunks store their two pieces in opposite order: no bank conflicts
                const uint32_t src[4] = {odd ? nope[i].z : nope[i].x, odd ? nope[i].w : nope[i].y,
                                         odd ? nope[i].x : nope[i].z, odd ? nope[i].y : nope[i].w};
                uint32_t d[8];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    e4m3_as_bf16(src[k], d[2 * k], d[2 * k + 1]);
                    d[2 * k] = mul_bf16x2(d[2 * k], f);
                    d[2 * k + 1] = mul_bf16x2(d[2 * k + 1], f);
                }
                if (__any_sync(0xffffffffu, e > 134u)) {
                    // (255, no number in UE8M0, makes infinity here as in the fp32 kernel)
                    const __nv_bfloat162 f2 = pow2_bf16x2(e == 255u ? 255u : e > 134u ? min(e - 134u, 127u) + 127u : 127u);
#pragma unroll
                    for (int k = 0; k < 8; ++k) d[k] = mul_bf16x2(d[k], f2);
                }
                if (lane < X_NOPE / 16) {
                    uint8_t* chunk = sm + XK_OFF + bk * XK_CHUNK;
                    const uint32_t row = (uint32_t)token_of(i), pc = 2u * (lane & 3) + (odd ? 1u : 0u);
                    *reinterpret_cast<uint4*>(chunk + xswz(row, pc)) = make_uint4(d[0], d[1], d[2], d[3]);
                    *reinterpret_cast<uint4*>(chunk + xswz(row, pc ^ 1u)) = make_uint4(d[4], d[5], d[6], d[7]);
                }
            }
            if (!ok) break;
#pragma unroll
            for (int u = 0; u < X_RPW / 4; ++u)
                *reinterpret_cast<uint4*>(sm + XK_OFF + 7 * XK_CHUNK + xswz((uint32_t)token_of((lane >> 3) + 4 * u), (uint32_t)lane & 7u)) = rp[u];
            if (lane == 0) sm[XV_OFF + (it & 1u) * X_G_WARPS + g] = (uint8_t)vbits;
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(XB_KFULL));
            load_rows(idx, extra_now);
            asm volatile("" : "+r"(idx_after));             // the index is first looked at here, not where it was asked for
            prefetch_rows(idx_after, extra);
            idx = idx_after;
            extra_now = extra;
            have = have_next;
            have_next = have_after;
        }
    } else if (warp == X_MMA_WARP) {
        // =================================================================== MMA issue
        const uint32_t k_lo = desc_lo(base + XK_OFF, 16), q_lo = desc_lo(base + XQ_OFF, 16);
        const uint32_t v_lo = desc_lo(base + XK_OFF, XK_CHUNK);       // MN-major: the next 64 dims lie a chunk further
        const uint32_t p_lo = desc_lo(base + XP_OFF, 16);
        uint32_t it = 0, rq = 0;
        bool ok = true;
        for (int req = meta.begin_req; req <= last_req && ok; ++req) {
            Work w;
            if (!get_work(p, meta, req, w)) continue;
            const int nst = (w.nblk + 1) >> 1;
            ok = mbar_wait_lean(bar(XB_QREADY), rq & 1u, abort_addr, WX_QREADY);
            ++rq;
            for (int j = 0; j < nst && ok; ++j, ++it) {
                ok = mbar_wait_lean(bar(XB_KFULL), it & 1u, abort_addr, WX_KFULL);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
#pragma unroll 1
                    for (int kc = 0; kc < 8; ++kc) {
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            mma_f16(tmem + XT_S, make_desc(k_lo + ((kc * XK_CHUNK + k * 32) >> 4), X_DESC_HI),
                                    make_desc(q_lo + ((kc * XQ_CHUNK + k * 32) >> 4), X_DESC_HI), IDESC_S, (kc | k) != 0);
                    }
                    tc_commit(bar(XB_SREADY));
                }
                __syncwarp();
                ok = mbar_wait_lean(bar(XB_PREADY), it & 1u, abort_addr, WX_PREADY);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
#pragma unroll 1
                    for (int kq = 0; kq < 4; ++kq) {        // 32 tokens: their rows may be overwritten as soon as they have been read
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
#pragma unroll
                            for (int part = 0; part < 2; ++part) {
#pragma unroll
                                for (int b = 0; b < 4; ++b)
                                    mma_f16(tmem + XT_O + 64 * b, make_desc(v_lo + ((2 * b * XK_CHUNK + (2 * kq + k) * 2048) >> 4), X_DESC_HI),
                                            make_desc(p_lo + ((part * XP_BYTES + (2 * kq + k) * 2048) >> 4), X_DESC_HI), IDESC_O,
                                            (j | kq | k | part) != 0);
                            }
                        }
                        tc_commit(bar(XB_KFREE + kq));
                    }
                    tc_commit(bar(XB_PVDONE));
                }
                __syncwarp();
            }
        }
    }

    if (*abort_flag != 0) {        // a wait gave up: MMAs may still be in flight; give them time to finish
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
    if (warp == X_MMA_WARP) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

}  // namespace

int launch_attn_exact(const AttnParams& p, cudaStream_t stream) {
    if (p.num_tokens == 0) return 0;
    static std::atomic<bool> attr_set[64];
    static int sm_count[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return set_error(SMLA_E_SHAPE, "attn_exact_kernel: device ordinal %d not supported", dev);
    if (!attr_set[dev]) {
        cudaFuncAttributes fa;
        if (cudaFuncGetAttributes(&fa, attn_exact_kernel) != cudaSuccess || fa.numRegs != X_REGS_LAUNCH)
            return set_error(SMLA_E_DEVICE, "attn_exact_kernel: compiled with %d registers per thread, the warpgroup budgets assume %d",
                             fa.numRegs, X_REGS_LAUNCH);
        const cudaError_t e = cudaFuncSetAttribute(attn_exact_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)X_SMEM);
        if (e != cudaSuccess) return set_error((int)e, "attn_exact_kernel: cannot reserve %u bytes of shared memory: %s", X_SMEM,
                                               cudaGetErrorString(e));
        cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev);
        attr_set[dev] = true;
    }
    const int halves = (p.num_heads + X_HEADS - 1) / X_HEADS;
    const int most = sm_count[dev] / halves > 0 ? sm_count[dev] / halves : 1;
    const int parts = p.sched ? p.num_parts : (p.num_tokens < most ? p.num_tokens : most);
    const dim3 grid(parts, halves);
    launch_dependent(attn_exact_kernel, grid, dim3(X_THREADS), X_SMEM, stream, p);
    return check_launch("attn_exact_kernel");
}

}  // namespace smla

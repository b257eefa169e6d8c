// Causal prefill attention for sm_100a on the 5th-generation tensor cores (tcgen05 + tensor memory).
//
// What it computes: for every sequence b, query head h and row t,
//     O[b][t][h] = softmax_{u <= t}( Q[b][t][h] . K[b][u][h / G] * scale ) V[b][u][h / G]
// which is what the engine produces when it runs its single-token forward once per prompt token with
// kv_len = t + 1 (tools/infer.cpp:271-274, src/model/model.cpp:68, attn() of include/kernels_cpu.hpp:140-167).
// The engine has no S x S kernel of its own; the results are pinned by that row-by-row definition.
//
// Layouts (dense, head_dim = 128 or 64, 16-bit elements): Q, O [B][S][H][D]; K, V [B][S][Hkv][D] — the engine's
// cache layout [row][kv_head][head_dim] per sequence.
//
// Work item = two 128-row query tiles that share one K/V stream (two query heads of the same kv head at the
// same rows when the GQA group is even, else two consecutive row tiles of one head). Persistent, one CTA per SM: the
// items are dealt longest causal span first, back and forth over the CTAs (4 x 2048 rows: 1024 items, no CTA more than
// one item above another), and an item's loads and first score products run while the previous item's result is
// written: 196 -> 181 us in a burst (758 TFLOP/s causal; 209 us in a sustained loop under the power cap). 12 warps:
//   warps 0-3   softmax of tile 0: thread r owns query row r (tensor-memory lane r), no shuffles needed
//   warps 4-7   softmax of tile 1
//   warp  8     TMA producer: an item's Q tiles, then its K and V tiles (64 keys x 128 dims, 128-byte swizzle)
//               through a 4-stage ring with separate barriers for K and V
//   warp  9     one thread issues every tcgen05.mma: S_t = Q_t K^T (both operands in shared memory,
//               accumulator in tensor memory) and O_t += P_t V (P read from tensor memory, V from shared
//               memory as an MN-major operand), in the order PV_0(j), QK_0(j+2), PV_1(j), QK_1(j+2)
//   warps 10-11 idle (they only take part in the register re-allocation of their warpgroup)
// Tensor memory (512 columns): two score buffers of 64 columns per tile, then O_0 | O_1, 128 fp32 columns each. With two
// score buffers the softmax of block j+1 never waits for the products of block j: with one buffer of 128 keys a tile's
// softmax (~ 2 000 clocks) and its 24 MMAs (1 536) took turns. An m128n64k16 MMA takes 48 clocks (its shared-memory
// reads), so 128 keys cost 3 584 tensor clocks for both tiles instead of 3 072, which still is less than the turns.
// 4 x 2048 rows, 32/8 heads of 128, bf16: 220 -> 196 us before the CTAs were persistent.
// P overwrites S in place as packed 16-bit pairs in columns [0,32). Two ways to hand P to the tensor cores (template
// PMODE):
//   kPResidual  P in the input type plus its rounding residual in columns [32,64) and a second PV MMA: ~2^-17,
//               the mode that meets the parity tolerance on every row (the default).
//   kPInput     P rounded once to the input type (fp16: 2^-11, bf16: 2^-9 per element), one PV MMA.
// A and B of one MMA must have the same 16-bit format: an fp16 P against a bf16 V (the instruction descriptor has
// separate format fields) raises an illegal-instruction error on this part, so there is no such mode.
// Online softmax follows the engine's state merge (src/attention.cu:41-65): running maximum m, sum l,
// accumulator rescaled by exp(m_old - m_new); the rescale is skipped until the maximum has grown by more
// than 2^8, and the true l normalises at the end, so the result is unchanged.
//
// Every wait is bounded; on expiry the role records ATTN_STATUS_WAIT_TIMEOUT, stops, and the CTA still
// runs its common exit (final barrier, tensor-memory release).
#include <cuda.h>

#include <algorithm>

#include "attn_internal.cuh"
#include "ptx_sm100.cuh"
#include "tcgen05_sm100.cuh"
#include "tma_tile.cuh"

namespace b200 {
namespace {

using namespace tc;

constexpr int BM = 128;   // query rows per tile
constexpr int BN = 64;    // keys per block
// head_dim is 128 or 64 (template HDIM); shared memory is laid out for 128
constexpr int kThreads = 384;
constexpr uint32_t kSubTileBytes = BM * 64 * 2;        // [128 query rows][64 elements], 128-byte rows, swizzled
constexpr uint32_t kTileBytes = 2 * kSubTileBytes;     // 128 x 128 16-bit elements (head_dim 64 fills the first half)
constexpr uint32_t kKvSubBytes = BN * 64 * 2;          // the same of a key block
constexpr uint32_t kKvBytes = 2 * kKvSubBytes;
constexpr int kStages = 4;
constexpr uint32_t kTmemCols = 512;
#ifdef ATTN_TRACE
float* g_prefill_debug = nullptr;
#endif

struct PrefillParams {
    void* o;
    int32_t o_dtype;
    int32_t in_dtype;  // ATTN_DTYPE_F16 | ATTN_DTYPE_BF16
    uint32_t batch, seq, n_heads, n_kv_heads, group;
    uint32_t m_tiles;     // ceil(seq / 128)
    uint32_t heads_x;     // head pairs (or heads) per row-tile step
    uint32_t items;       // work items of two tiles
    uint32_t pair_heads;  // 1: tiles are heads (2*hp, 2*hp+1) at the same rows; 0: rows (2*mp, 2*mp+1) of one head
    float scale_log2;
    uint32_t* status;
#ifdef ATTN_TRACE
    float* debug;  // optional [128][128] dump of the first S tile of CTA (0,0,0)
#endif
};

enum : int { kPResidual = 0, kPInput = 1 };

// ---- barriers (8 bytes each) inside shared memory ----
enum {
    BAR_Q_FULL = 0,
    BAR_Q_EMPTY = 1,
    BAR_K_FULL = 2,                   // [kStages]
    BAR_V_FULL = BAR_K_FULL + kStages,
    BAR_K_EMPTY = BAR_V_FULL + kStages,
    BAR_V_EMPTY = BAR_K_EMPTY + kStages,
    BAR_S_FULL = BAR_V_EMPTY + kStages,
    // [tile][block parity]: scores are there, probabilities are there, the block's PV product is complete. Two barriers
    // each, because scores run two blocks ahead: a side may be one phase behind, which one parity bit cannot tell.
    BAR_P_FULL = BAR_S_FULL + 4,
    BAR_O_DONE = BAR_P_FULL + 4,
    BAR_COUNT = BAR_O_DONE + 4
};

constexpr uint32_t kSmemQ = 0;
constexpr uint32_t kSmemK = kSmemQ + 2 * kTileBytes;
constexpr uint32_t kSmemV = kSmemK + kStages * kKvBytes;
constexpr uint32_t kSmemStage = kSmemV + kStages * kKvBytes;   // per tile: [128 rows][128 B] output staging
constexpr uint32_t kStageTileBytes = 128 * 128;
constexpr uint32_t kSmemBars = kSmemStage + 2 * kStageTileBytes;
constexpr uint32_t kSmemTmemPtr = kSmemBars + BAR_COUNT * 8;
constexpr uint32_t kSmemTotal = kSmemTmemPtr + 16;
constexpr uint32_t kSmemAlloc = kSmemTotal + 1024;  // slack to align the base to 1024 bytes

// ---- tensor-memory stores (the other wrappers are in tcgen05_sm100.cuh) ----
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&u)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
        "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(u[8]),
          "r"(u[9]), "r"(u[10]), "r"(u[11]), "r"(u[12]), "r"(u[13]), "r"(u[14]), "r"(u[15]), "r"(u[16]), "r"(u[17]),
          "r"(u[18]), "r"(u[19]), "r"(u[20]), "r"(u[21]), "r"(u[22]), "r"(u[23]), "r"(u[24]), "r"(u[25]), "r"(u[26]),
          "r"(u[27]), "r"(u[28]), "r"(u[29]), "r"(u[30]), "r"(u[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&u)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(u[8]),
          "r"(u[9]), "r"(u[10]), "r"(u[11]), "r"(u[12]), "r"(u[13]), "r"(u[14]), "r"(u[15])
        : "memory");
}

// Packed 16-bit pair -> two floats (exact).
template <bool BF16>
__device__ __forceinline__ void unpack2(uint32_t u, float& a, float& b) {
    if constexpr (BF16) {
        a = __uint_as_float(u << 16);
        b = __uint_as_float(u & 0xffff0000u);
    } else {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u));
        a = f.x;
        b = f.y;
    }
}

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Two fp32 operations per instruction.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack_f32x2(float a, float b) {
    f32x2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ void unpack_f32x2(f32x2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 fma_f32x2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 add_f32x2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ void report_timeout(uint32_t* status) {
    if (status) atomicOr(status, ATTN_STATUS_WAIT_TIMEOUT);
}

struct Item {
    uint32_t b, head[2], m0[2], nblk[2], n_iter;  // n_iter = key blocks of the longer tile
};

template <bool BF16, int PMODE, int HDIM>
__global__ void __launch_bounds__(kThreads, 1)
prefill_causal_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                      const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o,
                      const __grid_constant__ PrefillParams p) {
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* smem = smem_raw + (base - raw);
    const uint32_t bars = base + kSmemBars;
    auto bar = [&](int i) { return bars + 8u * i; };
    volatile uint32_t* tmem_ptr_smem = reinterpret_cast<volatile uint32_t*>(smem + kSmemTmemPtr);

    const int tid = threadIdx.x;
    const int warp = uniform_warp();
    const int lane = tid & 31;
    constexpr int HD = HDIM;
    constexpr uint32_t kLoadQ = (HD / 64) * kSubTileBytes, kLoadKv = (HD / 64) * kKvSubBytes;  // bytes of a tile actually loaded

    // ---- work items: two tiles each, dealt longest causal span first, back and forth over the CTAs ----
    const uint32_t nblk_total = (p.seq + BN - 1) / BN;
    auto item_of = [&](uint32_t round, Item& w) {
        const uint32_t pos = (round & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
        const uint32_t idx = round * gridDim.x + pos;
        if (idx >= p.items) return false;
        const uint32_t per_span = p.heads_x * p.batch;
        const uint32_t z = idx / per_span, rest = idx - z * per_span;
        w.b = rest / p.heads_x;
        const uint32_t x = rest - w.b * p.heads_x;
        if (p.pair_heads) {
            w.head[0] = 2 * x;
            w.head[1] = 2 * x + 1;
            w.m0[0] = w.m0[1] = (p.m_tiles - 1 - z) * BM;
        } else {
            const uint32_t mp = (p.m_tiles + 1) / 2 - 1 - z;
            w.head[0] = w.head[1] = x;
            w.m0[0] = 2 * mp * BM;
            w.m0[1] = w.m0[0] + BM;
        }
#pragma unroll
        for (int t = 0; t < 2; ++t) w.nblk[t] = w.m0[t] < p.seq ? min(nblk_total, (w.m0[t] + BM) / BN) : 0u;
        w.n_iter = max(w.nblk[0], w.nblk[1]);
        return true;
    };

    // ---- set-up: barriers, tensor memory ----
    if (tid == 0) {
        mbar_init(bar(BAR_Q_FULL), 1);
        mbar_init(bar(BAR_Q_EMPTY), 1);
        for (int s = 0; s < kStages; ++s) {
            mbar_init(bar(BAR_K_FULL + s), 1);
            mbar_init(bar(BAR_V_FULL + s), 1);
            mbar_init(bar(BAR_K_EMPTY + s), 1);
            mbar_init(bar(BAR_V_EMPTY + s), 1);
        }
        for (int t = 0; t < 2; ++t) {
            mbar_init(bar(BAR_S_FULL + 2 * t), 1);
            mbar_init(bar(BAR_S_FULL + 2 * t + 1), 1);
            mbar_init(bar(BAR_P_FULL + 2 * t), 128);
            mbar_init(bar(BAR_P_FULL + 2 * t + 1), 128);
            mbar_init(bar(BAR_O_DONE + 2 * t), 1);
            mbar_init(bar(BAR_O_DONE + 2 * t + 1), 1);
        }
        mbar_init_fence();
    }
    if (warp == 8) {
        tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_ptr_smem)), kTmemCols);
        tmem_relinquish();
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem_base = *tmem_ptr_smem;
    auto tmem_s = [&](int t, uint32_t buf) { return tmem_base + static_cast<uint32_t>(t) * 128u + buf * 64u; };
    auto tmem_o = [&](int t) { return tmem_base + 256u + static_cast<uint32_t>(t) * 128u; };

    if (warp < 8) {
        // =============================== softmax warpgroups ===============================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
        const int t = warp >> 2;                       // tile
        const int r = ((warp & 3) << 5) | lane;        // row inside the tile = tensor-memory lane
        const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) << 5) << 16;
        bool ok = true;
        uint32_t g0 = 0;  // key blocks of this tile before the current item: buffer and barrier phases run on over the items
        Item w;
        for (uint32_t round = 0; ok && item_of(round, w); ++round) {
        const uint32_t my_m0 = t ? w.m0[1] : w.m0[0], my_head = t ? w.head[1] : w.head[0], my_nblk = t ? w.nblk[1] : w.nblk[0];
        const uint32_t q_row = my_m0 + r;              // row index inside the sequence
        float m_used = -INFINITY;                      // maximum the stored probabilities are relative to (log2 units)
        float l = 0.f;
        for (uint32_t j = 0; j < my_nblk && ok; ++j) {
            const uint32_t g = g0 + j, buf = g & 1, par = (g >> 1) & 1;
            const uint32_t s_tmem = tmem_s(t, buf) + lane_addr;
            if (!mbar_wait(bar(BAR_S_FULL + 2 * t + buf), par)) { report_timeout(p.status); ok = false; break; }
            fence_after();
            float s[BN];
#pragma unroll
            for (int c = 0; c < BN / 32; ++c) {
                tmem_ld32(s_tmem + c * 32, *reinterpret_cast<float(*)[32]>(&s[c * 32]));
            }
            tmem_wait_ld();
#ifdef ATTN_TRACE
            if (p.debug && w.b == 0 && my_head == 0 && my_m0 == 0 && t == 0 && j < 2) {
#pragma unroll
                for (int c = 0; c < BN; ++c) p.debug[r * 128 + j * BN + c] = s[c];
            }
#endif
            // causal mask: only the diagonal blocks need it (keys of later blocks are never visited)
            if (j * BN + BN - 1 > q_row) {
#pragma unroll
                for (int c = 0; c < BN; ++c) {
                    if (j * BN + c > q_row) s[c] = -INFINITY;
                }
            }
            // four independent chains of three-input maxima
            float mx4[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) mx4[i] = max3(s[i], s[4 + i], s[8 + i]);
#pragma unroll
            for (int c = 12; c + 8 <= BN; c += 8) {
#pragma unroll
                for (int i = 0; i < 4; ++i) mx4[i] = max3(mx4[i], s[c + i], s[c + 4 + i]);
            }
            float mx = max3(fmaxf(mx4[0], mx4[1]), mx4[2], mx4[3]);
#pragma unroll
            for (int c = 12 + (BN - 12) / 8 * 8; c < BN; ++c) mx = fmaxf(mx, s[c]);
            mx *= p.scale_log2;
            // Rescale only when the maximum grew by more than 8 (probabilities stay below 2^8).
            float factor = 1.f;
            if (mx > m_used + 8.f) {
                factor = fast_exp2(m_used - mx);  // 0 on the first block (m_used = -inf)
                m_used = mx;
            }
            // Products of earlier blocks: the scores of block j were issued behind PV(j-2), so that one is over (waiting
            // for every phase in turn keeps the parities unambiguous); PV(j-1) may still be running and is
            // waited for only when O has to be rescaled.
            if (g >= 2 && !mbar_wait(bar(BAR_O_DONE + 2 * t + buf), par ^ 1)) { report_timeout(p.status); ok = false; break; }
            if (j > 0 && __any_sync(0xffffffffu, factor != 1.f)) {
                if (!mbar_wait(bar(BAR_O_DONE + 2 * t + (buf ^ 1)), ((g - 1) >> 1) & 1)) { report_timeout(p.status); ok = false; break; }
                fence_after();
#pragma unroll
                for (int c = 0; c < HD / 32; ++c) {
                    float o[32];
                    tmem_ld32(tmem_o(t) + lane_addr + c * 32, o);
                    tmem_wait_ld();
                    uint32_t u[32];
#pragma unroll
                    for (int i = 0; i < 32; ++i) u[i] = __float_as_uint(o[i] * factor);
                    tmem_st32(tmem_o(t) + lane_addr + c * 32, u);
                }
            }
            l *= factor;
            // probabilities; P overwrites S in place (every S value of this row is already in registers). Pairs of
            // elements share one packed fp32 instruction (scale, residual, sum).
            const f32x2 scale2 = pack_f32x2(p.scale_log2, p.scale_log2), m2 = pack_f32x2(-m_used, -m_used);
            const f32x2 minus1 = pack_f32x2(-1.f, -1.f);
            f32x2 sum2[2] = {pack_f32x2(0.f, 0.f), pack_f32x2(0.f, 0.f)};
#pragma unroll
            for (int c = 0; c < BN / 32; ++c) {
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    float p0, p1;
                    unpack_f32x2(fma_f32x2(pack_f32x2(s[c * 32 + 2 * i], s[c * 32 + 2 * i + 1]), scale2, m2), p0, p1);
                    p0 = fast_exp2(p0);
                    p1 = fast_exp2(p1);
                    const f32x2 pp = pack_f32x2(p0, p1);
                    sum2[i & 1] = add_f32x2(sum2[i & 1], pp);
                    // Rounded pair by one packed convert; its fp32 value is recovered with integer / half-add
                    // operations so that no scalar convert (special-function pipe, already busy with exp2) is used.
                    hi[i] = pack2<BF16>(p0, p1);
                    if constexpr (PMODE == kPResidual) {
                        float h0, h1;
                        unpack2<BF16>(hi[i], h0, h1);
                        float r0, r1;
                        unpack_f32x2(fma_f32x2(pack_f32x2(h0, h1), minus1, pp), r0, r1);
                        lo[i] = pack2<BF16>(r0, r1);
                    }
                }
                // 32 keys -> 16 packed columns: rounded part at column 16c, residual at BN / 2 + 16c
                tmem_st16(s_tmem + c * 16, hi);
                if constexpr (PMODE == kPResidual) tmem_st16(s_tmem + BN / 2 + c * 16, lo);
            }
            float s0, s1;
            unpack_f32x2(add_f32x2(sum2[0], sum2[1]), s0, s1);
            l += s0 + s1;
            tmem_wait_st();
            fence_before();
            mbar_arrive(bar(BAR_P_FULL + 2 * t + buf));
        }
        g0 += my_nblk;
        // ---- epilogue: O / l -> global ----
        if (ok && my_nblk > 0) {
            if (!mbar_wait(bar(BAR_O_DONE + 2 * t + ((g0 - 1) & 1)), ((g0 - 1) >> 1) & 1)) {
                report_timeout(p.status);
                ok = false;
            } else {
                fence_after();
                const float inv = l > 0.f ? 1.f / l : 0.f;
                // The tile leaves through shared memory and the TMA engine, 128 bytes of every row per pass: each
                // thread writes its row's 16-byte chunks XOR-swizzled by the row (the 128-byte swizzle the tensor
                // map expects; no bank conflicts), the four warps of the tile meet, and one thread issues the bulk
                // store, which also clips rows past the end of the sequence. Plain per-thread global stores (rows
                // are 8 KB apart) would sit in the load/store queue that this SM's MMA and TMA instructions also
                // pass through and stall them while they drain.
                const uint32_t stage = base + kSmemStage + t * kStageTileBytes;
                const bool f32_out = p.o_dtype == ATTN_DTYPE_F32;
                const int passes = f32_out ? HD / 32 : HD / 64;
#pragma unroll
                for (int pass = 0; pass < 4; ++pass) {
                    if (pass < passes) {
                        // 32 accumulator columns at a time (fp32 out: one pass; 16-bit out: half a pass)
                        const int n_ld = f32_out ? 1 : 2;
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            if (h < n_ld) {
                                float o[32];
                                tmem_ld32(tmem_o(t) + lane_addr + (f32_out ? pass * 32 : pass * 64 + h * 32), o);
                                tmem_wait_ld();
#pragma unroll
                                for (int c = 0; c < (8 >> 1) * 2; ++c) {
                                    if (f32_out) {
                                        const uint4 v = make_uint4(__float_as_uint(o[c * 4] * inv), __float_as_uint(o[c * 4 + 1] * inv),
                                                                   __float_as_uint(o[c * 4 + 2] * inv), __float_as_uint(o[c * 4 + 3] * inv));
                                        const uint32_t addr = stage + r * 128 + ((c ^ (r & 7)) << 4);
                                        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
                                    } else if (c < 4) {
                                        uint4 v;
                                        if (p.o_dtype == ATTN_DTYPE_BF16) {
                                            v = make_uint4(pack2<true>(o[c * 8] * inv, o[c * 8 + 1] * inv), pack2<true>(o[c * 8 + 2] * inv, o[c * 8 + 3] * inv),
                                                           pack2<true>(o[c * 8 + 4] * inv, o[c * 8 + 5] * inv), pack2<true>(o[c * 8 + 6] * inv, o[c * 8 + 7] * inv));
                                        } else {
                                            v = make_uint4(pack2<false>(o[c * 8] * inv, o[c * 8 + 1] * inv), pack2<false>(o[c * 8 + 2] * inv, o[c * 8 + 3] * inv),
                                                           pack2<false>(o[c * 8 + 4] * inv, o[c * 8 + 5] * inv), pack2<false>(o[c * 8 + 6] * inv, o[c * 8 + 7] * inv));
                                        }
                                        const int chunk = h * 4 + c;
                                        const uint32_t addr = stage + r * 128 + ((chunk ^ (r & 7)) << 4);
                                        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
                                    }
                                }
                            }
                        }
                        fence_async_smem();
                        named_bar_sync(1 + t, 128);
                        if ((warp & 3) == 0 && lane == 0) {
                            tma_store_4d(&tm_o, stage, pass * (f32_out ? 32 : 64), my_m0, my_head, w.b);
                            tma_store_commit();
                            tma_store_wait_read();  // the staging tile may be overwritten after this
                        }
                        named_bar_sync(1 + t, 128);
                    }
                }
            }
        }
        }
        if ((warp & 3) == 0 && lane == 0) tma_store_wait_all();
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp == 8 && elect_one()) {
            // =============================== TMA producer ===============================
            uint32_t st = 0, phase = 0, it = 0;
            bool ok = true;
            Item w;
            for (uint32_t round = 0; ok && item_of(round, w); ++round) {
                // the query tiles are overwritten once every score product of the previous item has read them
                if (round > 0 && !mbar_wait(bar(BAR_Q_EMPTY), (round - 1) & 1)) { ok = false; break; }
                const uint32_t kvh = w.head[0] / p.group;
                mbar_arrive_expect_tx(bar(BAR_Q_FULL), ((w.nblk[0] > 0) + (w.nblk[1] > 0)) * kLoadQ);
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    if (w.nblk[t] == 0) continue;
                    const uint32_t dst = base + kSmemQ + t * kTileBytes;
                    tma_load_4d(dst, &tm_q, bar(BAR_Q_FULL), 0, w.m0[t], w.head[t], w.b);
                    if (HD > 64) tma_load_4d(dst + kSubTileBytes, &tm_q, bar(BAR_Q_FULL), 64, w.m0[t], w.head[t], w.b);
                }
                for (uint32_t j = 0; j < w.n_iter; ++j, ++it) {
                    if (it >= kStages && !mbar_wait(bar(BAR_K_EMPTY + st), phase ^ 1)) { ok = false; break; }
                    const uint32_t kdst = base + kSmemK + st * kKvBytes;
                    mbar_arrive_expect_tx(bar(BAR_K_FULL + st), kLoadKv);
                    tma_load_4d(kdst, &tm_k, bar(BAR_K_FULL + st), 0, j * BN, kvh, w.b);
                    if (HD > 64) tma_load_4d(kdst + kKvSubBytes, &tm_k, bar(BAR_K_FULL + st), 64, j * BN, kvh, w.b);
                    if (it >= kStages && !mbar_wait(bar(BAR_V_EMPTY + st), phase ^ 1)) { ok = false; break; }
                    const uint32_t vdst = base + kSmemV + st * kKvBytes;
                    mbar_arrive_expect_tx(bar(BAR_V_FULL + st), kLoadKv);
                    tma_load_4d(vdst, &tm_v, bar(BAR_V_FULL + st), 0, j * BN, kvh, w.b);
                    if (HD > 64) tma_load_4d(vdst + kKvSubBytes, &tm_v, bar(BAR_V_FULL + st), 64, j * BN, kvh, w.b);
                    if (++st == kStages) st = 0, phase ^= 1;
                }
            }
            if (!ok) report_timeout(p.status);
        } else if (warp == 9 && elect_one()) {
            // =============================== MMA issuer ===============================
            constexpr uint32_t fmt = BF16 ? 1u : 0u;
            constexpr uint32_t idesc_qk = instr_desc(fmt, fmt, 0, BM, BN);  // S: 128 rows x 64 keys
            constexpr uint32_t idesc_pv = instr_desc(fmt, fmt, 1, BM, HD);  // O: 128 rows x head_dim
            const uint64_t q_desc = smem_desc(base + kSmemQ, 16, 1024), k_desc = smem_desc(base + kSmemK, 16, 1024);
            const uint64_t v_desc = smem_desc(base + kSmemV, kKvSubBytes, 1024);
            // S_t = Q_t K^T: MMAs of K = 16 over head_dim; operands K-major, 128-byte swizzle, 8-row groups 1024 B apart
            // (descriptors count in 16 bytes)
            uint32_t g0[2] = {0, 0};  // key blocks of each tile before the current item
            auto issue_qk = [&](int t, uint32_t j, uint32_t st) {
                const uint32_t buf = (g0[t] + j) & 1;
                const uint64_t qa = q_desc + t * (kTileBytes / 16), ka = k_desc + st * (kKvBytes / 16);
                const uint32_t d = tmem_s(t, buf);
#pragma unroll
                for (int kc = 0; kc < HD / 16; ++kc) {
                    mma_ss(d, qa + (kc >> 2) * (kSubTileBytes / 16) + (kc & 3) * 2,
                           ka + (kc >> 2) * (kKvSubBytes / 16) + (kc & 3) * 2, idesc_qk, kc > 0);
                }
                commit(bar(BAR_S_FULL + 2 * t + buf));
            };
            // O_t += P_t V: MMAs of K = 16 keys; A = P in tensor memory (8 packed columns per MMA), B = V as an
            // MN-major operand: 64-dim halves one sub-tile apart (leading offset), 8-key groups 1024 B apart (stride)
            auto issue_pv = [&](int t, uint32_t j, uint32_t st) {
                const uint32_t buf = (g0[t] + j) & 1;
                const uint64_t va = v_desc + st * (kKvBytes / 16);
                const uint32_t pa = tmem_s(t, buf);
#pragma unroll
                for (int kc = 0; kc < BN / 16; ++kc) mma_ts(tmem_o(t), pa + kc * 8, va + kc * 128, idesc_pv, j > 0 || kc > 0);
                if constexpr (PMODE == kPResidual) {
#pragma unroll
                    for (int kc = 0; kc < BN / 16; ++kc) mma_ts(tmem_o(t), pa + BN / 2 + kc * 8, va + kc * 128, idesc_pv, 1);
                }
                commit(bar(BAR_O_DONE + 2 * t + buf));
            };
            // Scores run two blocks ahead of the products: Q K^T of block j + 2 is issued right behind P V of block j
            // (whose probabilities lie in the buffer it overwrites; the tensor pipe works in order).
            // An item's first two score products are issued behind the previous item's last product, while the softmax
            // warps still write that item's result.
            bool ok = true;
            uint32_t st = 0, phase = 0, kst = 0, kphase = 0;  // ring position of the next V block, of the next K block
            Item w;
            for (uint32_t round = 0; ok && item_of(round, w); ++round) {
                ok = mbar_wait(bar(BAR_Q_FULL), round & 1);
                auto next_k = [&]() {
                    if (++kst == kStages) kst = 0, kphase ^= 1;
                };
                for (uint32_t j = 0; j < 2 && j < w.n_iter && ok; ++j) {
                    ok = mbar_wait(bar(BAR_K_FULL + kst), kphase);
                    if (!ok) break;
                    fence_after();
#pragma unroll
                    for (int t = 0; t < 2; ++t)
                        if (j < w.nblk[t]) issue_qk(t, j, kst);
                    commit(bar(BAR_K_EMPTY + kst));
                    if (j + 1 == w.n_iter) commit(bar(BAR_Q_EMPTY));
                    next_k();
                }
                for (uint32_t j = 0; j < w.n_iter && ok; ++j) {
                    if (!mbar_wait(bar(BAR_V_FULL + st), phase)) { ok = false; break; }
                    const bool more = j + 2 < w.n_iter;
                    bool k_ready = false;
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        if (!ok || j >= w.nblk[t]) continue;
                        const uint32_t g = g0[t] + j;
                        if (!mbar_wait(bar(BAR_P_FULL + 2 * t + (g & 1)), (g >> 1) & 1)) { ok = false; break; }
                        fence_after();
                        issue_pv(t, j, st);
                        if (j + 2 < w.nblk[t]) {
                            if (!k_ready) {
                                if (!mbar_wait(bar(BAR_K_FULL + kst), kphase)) { ok = false; break; }
                                fence_after();
                                k_ready = true;
                            }
                            issue_qk(t, j + 2, kst);
                        }
                    }
                    if (!ok) break;
                    commit(bar(BAR_V_EMPTY + st));
                    if (++st == kStages) st = 0, phase ^= 1;
                    if (more) {
                        commit(bar(BAR_K_EMPTY + kst));
                        if (j + 3 == w.n_iter) commit(bar(BAR_Q_EMPTY));
                        next_k();
                    }
                }
                g0[0] += w.nblk[0];
                g0[1] += w.nblk[1];
            }
            if (!ok) report_timeout(p.status);
        }
    }

    // ---- common exit: everybody meets, then the allocating warp releases tensor memory ----
    fence_before();
    __syncthreads();
    if (warp == 8) {
        fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

// ------------------------------------------------------------------------------------------------ host
// [B][S][heads][head_dim] tensor viewed as (dim, row, head, batch); box = 128 bytes of box_rows rows, 128-byte swizzle.
int make_map(CUtensorMap* map, const void* ptr, int32_t dtype, uint32_t batch, uint32_t seq, uint32_t heads,
             uint32_t HD, uint32_t box_rows) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return ATTN_ERR_CUDA;
    const cuuint64_t esz = dtype == ATTN_DTYPE_F32 ? 4 : 2;
    const cuuint64_t dims[4] = {HD, seq, heads, batch};
    const cuuint64_t strides[3] = {static_cast<cuuint64_t>(heads) * HD * esz, static_cast<cuuint64_t>(HD) * esz,
                                   static_cast<cuuint64_t>(seq) * heads * HD * esz};
    const cuuint32_t box[4] = {static_cast<cuuint32_t>(128 / esz), box_rows, 1, 1};  // 128-byte rows
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUtensorMapDataType dt = dtype == ATTN_DTYPE_F32    ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                   : dtype == ATTN_DTYPE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                              : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    CUresult r = enc(map, dt,
                     4, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        g_last_cuda_error = static_cast<int>(r);
        return ATTN_ERR_CUDA;
    }
    return ATTN_OK;
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" int attn_prefill_causal(const AttnPrefillArgs* a, void* stream_v) {
    if (!a || !a->o || !a->q || !a->k || !a->v) return ATTN_ERR_INVALID_ARG;
    if (a->batch == 0 || a->seq_len == 0 || a->n_heads == 0 || a->n_kv_heads == 0) return ATTN_ERR_INVALID_ARG;
    if (a->n_heads % a->n_kv_heads != 0) return ATTN_ERR_INVALID_ARG;
    if (a->dtype != ATTN_DTYPE_F16 && a->dtype != ATTN_DTYPE_BF16) return ATTN_ERR_UNSUPPORTED;
    if (a->o_dtype != ATTN_DTYPE_F32 && a->o_dtype != a->dtype) return ATTN_ERR_UNSUPPORTED;
    if (a->head_dim != 128 && a->head_dim != 64) return ATTN_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(a->q) | reinterpret_cast<uintptr_t>(a->k) | reinterpret_cast<uintptr_t>(a->v) |
         reinterpret_cast<uintptr_t>(a->o)) & 15u)
        return ATTN_ERR_ALIGNMENT;
    DeviceInfo dev{};
    int rc = current_device_info(&dev);
    if (rc != ATTN_OK) return rc;
    if (dev.cc_major != 10) return ATTN_ERR_DEVICE;

    CUtensorMap tm_q, tm_k, tm_v, tm_o;
    if ((rc = make_map(&tm_o, a->o, a->o_dtype, a->batch, a->seq_len, a->n_heads, a->head_dim, BM)) != ATTN_OK) return rc;
    if ((rc = make_map(&tm_q, a->q, a->dtype, a->batch, a->seq_len, a->n_heads, a->head_dim, BM)) != ATTN_OK) return rc;
    if ((rc = make_map(&tm_k, a->k, a->dtype, a->batch, a->seq_len, a->n_kv_heads, a->head_dim, BN)) != ATTN_OK) return rc;
    if ((rc = make_map(&tm_v, a->v, a->dtype, a->batch, a->seq_len, a->n_kv_heads, a->head_dim, BN)) != ATTN_OK) return rc;

    PrefillParams p{};
    p.o = a->o;
    p.o_dtype = a->o_dtype;
    p.in_dtype = a->dtype;
    p.batch = a->batch;
    p.seq = a->seq_len;
    p.n_heads = a->n_heads;
    p.n_kv_heads = a->n_kv_heads;
    p.group = a->n_heads / a->n_kv_heads;
    p.m_tiles = (a->seq_len + BM - 1) / BM;
    p.pair_heads = (p.group % 2 == 0) ? 1u : 0u;
    const float scale = a->scale != 0.f ? a->scale : 1.0f / sqrtf(static_cast<float>(a->head_dim));
    p.scale_log2 = scale * 1.4426950408889634f;
    p.status = a->status;
#ifdef ATTN_TRACE
    p.debug = g_prefill_debug;
#endif
    if (a->p_mode > 1) return ATTN_ERR_INVALID_ARG;

    p.heads_x = p.pair_heads ? a->n_heads / 2 : a->n_heads;
    const uint64_t spans = p.pair_heads ? p.m_tiles : (p.m_tiles + 1) / 2;
    const uint64_t items = spans * p.heads_x * a->batch;
    if (items > 0x7fffffffull || a->batch > 65535u || spans > 65535u) return ATTN_ERR_UNSUPPORTED;
    p.items = static_cast<uint32_t>(items);
    const dim3 grid(static_cast<uint32_t>(std::min<uint64_t>(items, static_cast<uint64_t>(dev.sm_count))));
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    auto launch = [&](auto kernel) -> int {
        B200_CUDA_TRY(allow_max_smem(kernel));
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = grid;
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = kSmemAlloc;
        cfg.stream = stream;
        B200_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, tm_q, tm_k, tm_v, tm_o, p));
        g_launch_count.fetch_add(1, std::memory_order_relaxed);
        return ATTN_OK;
    };
    const bool single = a->p_mode == ATTN_PREFILL_P_INPUT_TYPE;
    if (a->head_dim == 128) {
        if (a->dtype == ATTN_DTYPE_BF16) {
            return single ? launch(prefill_causal_kernel<true, kPInput, 128>) : launch(prefill_causal_kernel<true, kPResidual, 128>);
        }
        return single ? launch(prefill_causal_kernel<false, kPInput, 128>) : launch(prefill_causal_kernel<false, kPResidual, 128>);
    }
    if (a->dtype == ATTN_DTYPE_BF16) {
        return single ? launch(prefill_causal_kernel<true, kPInput, 64>) : launch(prefill_causal_kernel<true, kPResidual, 64>);
    }
    return single ? launch(prefill_causal_kernel<false, kPInput, 64>) : launch(prefill_causal_kernel<false, kPResidual, 64>);
}

#ifdef ATTN_TRACE
// Profiling build only: [128][128] floats that receive the raw Q.K^T of the first key block of the last row tile of
// head 0 / sequence 0 of every following attn_prefill_causal call (null = off).
extern "C" void attn_trace_set_prefill_debug(float* s_tile) { g_prefill_debug = s_tile; }
#endif

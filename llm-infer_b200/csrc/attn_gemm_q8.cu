// Projection of many tokens at once by Q8_0 weights (the prompt phase of a Q8_0 model) on the 5th-generation tensor cores:
//
//     C[t][j] (+)= sum_b d[j][b] * ( sum_{i in block b} A[t][i] * q[j][i] )        t < m tokens, j < n_out, 32 i per block
//
// with A as the fp16 pair of attn_gemm_f16 (value + residual, ~ 22 bits) and the weight as it is stored: an int8 q, exact
// in fp16, and the fp16 scale d of its block of 32. The engine names the type only (include/gguf.hpp:28); per token this
// is its matmul() (include/kernels_cpu.hpp:69-80) over fp32(d) * q.
//
// Why a kernel of its own: as an fp16 pair (attn_gemm_pair) the weight d * q needs a residual matrix and every product
// three MMAs. q alone is exact, so two are enough; the price is that the sum of a block leaves the tensor cores after 32
// elements and is scaled and added in fp32 registers. The weights are the M side of the MMA (a tensor-memory lane = a weight
// row), so a thread needs ONE scale per block for all its tokens. The error falls too, because the tensor cores truncate the
// short sums only: 4.9e-6 -> 2.1e-7 at k = 4096, 1.7e-5 -> 3.8e-7 at 14336 (relative, against float64).
//
// Persistent; a tile is PARTS x 128 weight rows x up to 128 tokens per CTA, two CTAs share the token side (PAIR, tcgen05
// cta_group::2, M 256). 12 warps:
//   warp 0      TMA producer: PARTS weight tiles [128][64] and its share of the token tiles (value, residual), 128-byte
//               swizzle, a ring of 192 KB
//   warp 1      one thread issues, per block of 32 and part, residual and value MMAs (K 16 each) into one of four
//               accumulators of 128 columns, and hands it over
//   warps 4-11  thread = weight row = tensor-memory lane, a warpgroup per part (or half of the tile's tokens): reads the
//               block's sums, multiplies by the row's scale and adds (fma.rn.f32x2) into up to 128 registers; setmaxnreg gives
//               these warps 232. The next chunk's tcgen05.ld is in flight while a chunk is added.
// At the tile's end a warp stores 32 consecutive outputs of a token at a time. With `swiglu` the two parts are the gate rows
// and the matching up rows; their warpgroups exchange halves through shared memory and write silu(gate) * up as the fp16 pair.
// What bounds it: reading and adding the block sums (a wait, a vote and a hand-back per block and ~ 50 clocks per 16 columns
// keep the tensor pipe at about half), in a long prompt phase the power cap. Sustained, pair -> here: 9101 x 28672 x 4096 (SwiGLU)
// 4.60 -> 4.05 ms, 9101 x 4096 x 4096 655 -> 553 us, 1003 x 4096 x 4096 82 -> 64, 48 x 4096 x 14336 143 -> 92.
#include <algorithm>
#include <type_traits>

#include "attn_internal.cuh"
#include "tcgen05_sm100.cuh"
#include "tma_tile.cuh"

namespace b200 {
namespace {

using namespace tc;

constexpr int kRowsM = 128, kStepK = 64, kBlockK = 32;
constexpr int kMaxStages = 6;
constexpr int kAccWarps = 8;
constexpr int kThreads = (4 + kAccWarps) * 32;
constexpr uint32_t kWTile = kRowsM * kStepK * 2;  // 16 KB
constexpr uint32_t kRowBytes = kStepK * 2;        // one row of a tile
constexpr uint32_t kSmemLimit = 227 * 1024;
constexpr uint32_t kTailUsed = 256;               // barriers, tensor-memory address
constexpr uint32_t kTailBytes = kTailUsed + 1024; // ... and slack to align the base to 1024
constexpr uint32_t kExchangeBytes = 2 * 32 * kRowsM * 4;  // swiglu: 32 tokens of 128 rows in either direction
constexpr uint32_t kBufs = 4, kBufCols = 128;     // accumulators in tensor memory

struct Q8GemmParams {
    float* c;
    __half* out_hi;  // swiglu
    __half* out_lo;
    const __half* d;       // [w_rows][d_pitch]
    uint64_t ldc;
    uint32_t m, n_out, k;  // n_out: columns of the result (swiglu: the hidden dimension)
    uint32_t w_rows, d_pitch;
    uint32_t t_tiles, r_tiles, band;
    uint32_t stages;
    uint32_t swiglu;
    int32_t accumulate;
    uint32_t* status;
};

// tokens of a tile that one CTA loads
constexpr uint32_t tile_tokens(bool pair, uint32_t n_tile) { return pair ? n_tile / 2 : n_tile; }
constexpr uint32_t stage_bytes_of(bool pair, uint32_t parts, uint32_t n_tile) {
    return parts * kWTile + 2 * tile_tokens(pair, n_tile) * kRowBytes;
}

enum { B_FULL = 0, B_EMPTY = B_FULL + kMaxStages, B_ACC_FULL = B_EMPTY + kMaxStages, B_ACC_EMPTY = B_ACC_FULL + kBufs,
       B_XCHG = B_ACC_EMPTY + kBufs, B_BARS = B_XCHG + 1 };

// Tile t of the flat list: bands of `band` token tiles, inside a band the token tile varies fastest.
__device__ __forceinline__ void tile_of(const Q8GemmParams& p, uint32_t t, uint32_t& tt, uint32_t& rt) {
    const uint32_t per_band = p.band * p.r_tiles;
    const uint32_t b = t / per_band, r = t - b * per_band;
    const uint32_t rows = min(p.band, p.t_tiles - b * p.band);
    rt = r / rows;
    tt = b * p.band + (r - rt * rows);
}

// First weight row of one part of a row tile for one CTA of the pair.
template <bool PAIR, int PARTS>
__device__ __forceinline__ uint32_t part_row(const Q8GemmParams& p, uint32_t rt, int part, uint32_t rank) {
    constexpr uint32_t kSpan = kRowsM * (PAIR ? 2 : 1);  // rows of one part over the pair
    const uint32_t base = p.swiglu ? rt * kSpan + part * p.n_out : (rt * PARTS + part) * kSpan;
    return base + rank * kRowsM;
}

// c0 += a0 * s, c1 += a1 * s in one instruction. (The pairs are packed inside the asm: with 64-bit accumulators the compiler
// moved them around at the loop's back edge, 9101 x 28672 x 4096 4.24 -> 3.98 ms.)
__device__ __forceinline__ void fma_pair(float& c0, float& c1, uint32_t a0, uint32_t a1, float s) {
    asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\tmov.b64 c, {%0, %1};\n\t"
        "fma.rn.f32x2 c, a, b, c;\n\tmov.b64 {%0, %1}, c;\n\t}"
        : "+f"(c0), "+f"(c1)
        : "r"(a0), "r"(a1), "f"(s));
}
// 16 columns of this thread's tensor-memory lane.
__device__ __forceinline__ void ld_chunk(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
// The wait for this thread's tensor-memory loads, tied to the registers they fill: arithmetic on them stays behind it.
template <int N>
__device__ __forceinline__ void wait_ld(uint32_t (&r)[N]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < N; ++i) asm volatile("" : "+r"(r[i]));
}

template <bool PAIR, int PARTS, int N_TILE>
__global__ void __launch_bounds__(kThreads, 1)
gemm_q8_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_hi,
               const __grid_constant__ CUtensorMap tm_lo, const __grid_constant__ Q8GemmParams p) {
    constexpr uint32_t kStageBytes = stage_bytes_of(PAIR, PARTS, N_TILE);
    constexpr uint32_t kTok = tile_tokens(PAIR, N_TILE), kTokBytes = kTok * kRowBytes;
    constexpr int COLS = PARTS == 2 ? N_TILE : N_TILE / 2;  // tokens of a tile per thread: all of one part, or half of the only one
    constexpr int CH = 16;                                  // columns per tensor-memory load
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;  // swizzled tiles want 1024-byte alignment
    unsigned char* smem = smem_raw + (base - raw);
    const uint32_t bars_at = p.stages * kStageBytes;
    const uint32_t bars = base + bars_at;
    auto bar = [&](int i) { return bars + 8u * i; };
    volatile uint32_t* tmem_ptr_smem = reinterpret_cast<volatile uint32_t*>(smem + bars_at + B_BARS * 8);

    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const uint32_t rank = PAIR ? cluster_rank() : 0u;
    const uint32_t worker = PAIR ? blockIdx.x / 2 : blockIdx.x, workers = PAIR ? gridDim.x / 2 : gridDim.x;
    const uint32_t tiles = p.t_tiles * p.r_tiles, k_steps = p.k / kStepK;

    if (tid == 0) {
        for (uint32_t s = 0; s < p.stages; ++s) {
            mbar_init(bar(B_FULL + s), 1);
            mbar_init(bar(B_EMPTY + s), 1);
        }
        for (uint32_t a = 0; a < kBufs; ++a) {
            mbar_init(bar(B_ACC_FULL + a), 1);
            mbar_init(bar(B_ACC_EMPTY + a), kAccWarps / PARTS * (PAIR ? 2 : 1));  // one arrival per reading warp
        }
        mbar_init(bar(B_XCHG), kAccWarps);
        mbar_init_fence();
    }
    if (warp == 1) {
        if constexpr (PAIR) {
            tmem_alloc_pair(smem_u32(const_cast<uint32_t*>(tmem_ptr_smem)), 512);
            tmem_relinquish_pair();
        } else {
            tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_ptr_smem)), 512);
            tmem_relinquish();
        }
    }
    fence_before();
    __syncthreads();
    if constexpr (PAIR) cluster_sync();  // the partner's barriers exist before anything is counted on them
    fence_after();
    const uint32_t tmem_base = *tmem_ptr_smem;

    grid_dep_launch_dependents();
    grid_dep_wait();

    if (warp < 4) {
        // (40 + 2 x 232) x 128 registers = the 168 x 384 that the block was launched with
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == 0 && elect_one()) {
            // =============================== TMA producer ===============================
            constexpr uint32_t bytes = PARTS * kWTile + 2 * kTokBytes;
            uint32_t it = 0, s = 0, phase = 0;
            bool ok = true;
            for (uint32_t t = worker; t < tiles && ok; t += workers) {
                uint32_t tt, rt;
                tile_of(p, t, tt, rt);
                const int tok = static_cast<int>(tt * N_TILE + rank * kTok);
                for (uint32_t ks = 0; ks < k_steps; ++ks, ++it) {
                    if (it >= p.stages && !mbar_wait(bar(B_EMPTY + s), phase ^ 1)) {
                        if (p.status) atomicOr(p.status, ATTN_STATUS_WAIT_TIMEOUT);
                        ok = false;
                        break;
                    }
                    const uint32_t dst = base + s * kStageBytes;
                    const uint32_t full = bar(B_FULL + s);
                    const int kc = static_cast<int>(ks * kStepK);
                    auto load = [&](uint32_t at, const CUtensorMap* map, int row) {
                        if constexpr (PAIR) tma_load_2d_pair(dst + at, map, full, kc, row);
                        else tma_load_2d(dst + at, map, full, kc, row);
                    };
                    if (rank == 0) mbar_arrive_expect_tx(full, PAIR ? 2 * bytes : bytes);
#pragma unroll
                    for (int part = 0; part < PARTS; ++part)
                        load(part * kWTile, &tm_w, static_cast<int>(part_row<PAIR, PARTS>(p, rt, part, rank)));
                    load(PARTS * kWTile, &tm_hi, tok);
                    load(PARTS * kWTile + kTokBytes, &tm_lo, tok);
                    if (++s == p.stages) s = 0, phase ^= 1;
                }
            }
        } else if (warp == 1 && rank == 0 && elect_one()) {
            // =============================== MMA issuer ===============================
            constexpr uint32_t idesc = instr_desc(0, 0, 0, PAIR ? 2 * kRowsM : kRowsM, N_TILE);
            auto mma = [&](uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
                if constexpr (PAIR) mma_ss_pair(d, a, b, idesc, acc);
                else mma_ss(d, a, b, idesc, acc);
            };
            auto done = [&](uint32_t b) {
                if constexpr (PAIR) commit_pair(b);
                else commit(b);
            };
            const uint64_t desc0 = smem_desc(base, 16, 1024);
            uint32_t s = 0, phase = 0, buf = 0, use = 0;  // accumulator and how often it was used before
            bool ok = true, ready = true;                 // ready: the accumulator was seen free while the last MMAs were issued
            for (uint32_t t = worker; t < tiles && ok; t += workers) {
                for (uint32_t ks = 0; ks < k_steps && ok; ++ks) {
                    if (!mbar_wait(bar(B_FULL + s), phase)) {
                        if (p.status) atomicOr(p.status, ATTN_STATUS_WAIT_TIMEOUT);
                        ok = false;
                        break;
                    }
                    // K-major operands, 128-byte swizzle: 32 bytes per k-step of 16, 8-row groups 1024 bytes apart
                    const uint64_t w0 = desc0 + s * (kStageBytes / 16);
                    const uint64_t hi0 = w0 + PARTS * (kWTile / 16), lo0 = hi0 + kTokBytes / 16;
#pragma unroll
                    for (int u = 0; u < 2 * PARTS; ++u) {
                        const int blk = u / PARTS, part = u % PARTS;
                        if (!ready && !mbar_wait(bar(B_ACC_EMPTY + buf), (use - 1) & 1)) {
                            if (p.status) atomicOr(p.status, ATTN_STATUS_WAIT_TIMEOUT);
                            ok = false;
                            break;
                        }
                        fence_after();
                        const uint32_t d = tmem_base + buf * kBufCols, full = bar(B_ACC_FULL + buf);
                        // (a look at a barrier takes ~ 100 clocks next to the MMAs' operand reads: it is under way while these
                        // four are issued)
                        if (++buf == kBufs) buf = 0, ++use;
                        ready = use == 0 || mbar_test(bar(B_ACC_EMPTY + buf), (use - 1) & 1);
                        const uint64_t w = w0 + part * (kWTile / 16) + 4 * blk;
                        mma(d, w, lo0 + 4 * blk, 0);          // residuals first: the small sums are added up first
                        mma(d, w + 2, lo0 + 4 * blk + 2, 1);
                        mma(d, w, hi0 + 4 * blk, 1);
                        mma(d, w + 2, hi0 + 4 * blk + 2, 1);
                        // one commit per accumulator and none of its own for the stage, which a scaling warp hands back when it
                        // sees the last accumulator of the stage
                        done(full);
                    }
                    if (++s == p.stages) s = 0, phase ^= 1;
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
        // =============================== scale and add ===============================
        const uint32_t quarter = warp & 3, group = (warp - 4) >> 2;
        const int part = PARTS == 2 ? static_cast<int>(group) : 0;
        const uint32_t col0 = PARTS == 2 ? 0u : group * COLS;
        const uint32_t lane_addr = tmem_base + ((quarter * 32) << 16) + col0;
        constexpr int CHUNKS = COLS / CH;
        constexpr uint32_t kNextBuf = PARTS == 2 ? 2 : 1;  // from a block's accumulator to the next block's
        const uint32_t n_pairs = p.k / (2 * kBlockK);
        uint32_t empty0 = bar(B_ACC_EMPTY);                // the leader's, also for its partner
        if constexpr (PAIR) empty0 = cluster_address(empty0, 0);
        uint32_t first = part, phase = 0;                  // accumulator of a pair's first block, parity of its barrier
        uint32_t exchanges = 0, stage = 0;
        bool ok = true;
        // The votes let all lanes of the warp give up or go on.
        auto wait_warp = [&](uint32_t b, uint32_t parity) {
            if (!__all_sync(0xffffffffu, mbar_try_wait(b, parity)) && !__all_sync(0xffffffffu, mbar_wait(b, parity))) {
                if (lane == 0 && p.status) atomicOr(p.status, ATTN_STATUS_WAIT_TIMEOUT);
                ok = false;
            }
        };
        for (uint32_t t = worker; t < tiles && ok; t += workers) {
            uint32_t tt, rt;
            tile_of(p, t, tt, rt);
            const uint32_t row = part_row<PAIR, PARTS>(p, rt, part, rank) + quarter * 32 + lane;
            // (rows past the matrix: zeros from TMA, any scale; the pitch covers whole groups of eight blocks)
            const uint4* dsrc = reinterpret_cast<const uint4*>(p.d + static_cast<size_t>(min(row, p.w_rows - 1)) * p.d_pitch);
            // the scales of four pairs of blocks, and the next four on their way (moved only when they are due: a move out of the
            // register that a load is filling waits for the load)
            uint4 dq, dnext = __ldg(dsrc);
            float acc[COLS];
#pragma unroll
            for (int i = 0; i < COLS; ++i) acc[i] = 0.f;
#pragma unroll 1
            for (uint32_t pb = 0; pb < n_pairs; ++pb) {
                if ((pb & 3) == 0) {
                    dq = dnext;
                    if (pb + 4 < n_pairs) dnext = __ldg(dsrc + pb / 4 + 1);
                }
                const float2 sc = __half22float2(*reinterpret_cast<const __half2*>(&dq.x));  // of the two blocks
                dq.x = dq.y, dq.y = dq.z, dq.z = dq.w;
                // (no load is in flight over the loop's back edge, where the compiler may copy registers)
                uint32_t v[2][CH];
                wait_warp(bar(B_ACC_FULL + first), phase);
                if (!ok) break;
                fence_after();
                ld_chunk(lane_addr + first * kBufCols, v[0]);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const uint32_t buf = first + u * kNextBuf;
                    const float scale = u ? sc.y : sc.x;
#pragma unroll
                    for (int c = 0; c < CHUNKS; ++c) {
                        const int at = (u * CHUNKS + c) & 1;
                        wait_ld(v[at]);
                        if (c < CHUNKS - 1) {
                            ld_chunk(lane_addr + buf * kBufCols + (c + 1) * CH, v[at ^ 1]);
                        } else {
                            // this accumulator is read: hand it back, and start on the next one
                            fence_before();
                            __syncwarp();
                            if (lane == 0) {
                                if constexpr (PAIR) mbar_arrive_cluster_relaxed(empty0 + 8 * buf);
                                else mbar_arrive(empty0 + 8 * buf);
                            }
                            if (u == 0) {
                                wait_warp(bar(B_ACC_FULL + buf + kNextBuf), phase);
                                if (warp == 8) {  // the last accumulator of the stage: its operands have been read
                                    if (lane == 0) mbar_arrive(bar(B_EMPTY + stage));
                                    if (++stage == p.stages) stage = 0;
                                }
                                fence_after();
                                ld_chunk(lane_addr + (buf + kNextBuf) * kBufCols, v[at ^ 1]);
                            }
                        }
#pragma unroll
                        for (int i = 0; i < CH; i += 2) fma_pair(acc[c * CH + i], acc[c * CH + i + 1], v[at][i], v[at][i + 1], scale);
                    }
                }
                if (PARTS == 2 || first != 0) phase ^= 1;
                if (PARTS == 1) first ^= 2;
                if (!ok) break;
            }
            if (!ok) break;
            const uint32_t tok0 = tt * N_TILE + col0;
            if (p.swiglu) {
                if constexpr (PARTS == 2) {
                    // Gate and up values of one output lie in two warps. In rounds of 64 tokens each side hands the other half
                    // of its values over through shared memory and finishes the other half itself.
                    float* s_x = reinterpret_cast<float*>(smem + bars_at + kTailUsed);
                    const uint32_t r128 = quarter * 32 + lane;
                    const uint32_t hid = row - part * p.n_out;
#pragma unroll
                    for (int r = 0; r < N_TILE / 64; ++r) {
                        float* mine = s_x + (group ^ 1) * (32 * kRowsM) + r128;  // read by the other side
                        const float* theirs = s_x + group * (32 * kRowsM) + r128;
                        // side 0 (gate) finishes the round's first 32 tokens, side 1 (up) the last 32
                        if (group == 0) {
#pragma unroll
                            for (int i = 0; i < 32; ++i) mine[i * kRowsM] = acc[r * 64 + 32 + i];
                        } else {
#pragma unroll
                            for (int i = 0; i < 32; ++i) mine[i * kRowsM] = acc[r * 64 + i];
                        }
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar(B_XCHG));
                        wait_warp(bar(B_XCHG), exchanges++ & 1);
                        if (!ok) break;
                        if (hid < p.n_out) {
                            const uint32_t tk = tok0 + r * 64 + group * 32;
                            size_t o = static_cast<size_t>(tk) * p.n_out + hid;
                            auto finish = [&](int i, float gate, float up) {
                                // silu(x) = x / (1 + expf(-x)), src/model/block.cpp:206-210
                                float x = __fdiv_rn(gate, 1.0f + expf(-gate)) * up;
                                x = fminf(fmaxf(x, -65504.f), 65504.f);
                                const __half hi = __float2half_rn(x);
                                if (tk + i < p.m) {
                                    p.out_hi[o] = hi;
                                    p.out_lo[o] = __float2half_rn(x - __half2float(hi));
                                }
                                o += p.n_out;
                            };
                            if (group == 0) {
#pragma unroll
                                for (int i = 0; i < 32; ++i) finish(i, acc[r * 64 + i], theirs[i * kRowsM]);
                            } else {
#pragma unroll
                                for (int i = 0; i < 32; ++i) finish(i, theirs[i * kRowsM], acc[r * 64 + 32 + i]);
                            }
                        }
                        // both sides have read before either writes again
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar(B_XCHG));
                        wait_warp(bar(B_XCHG), exchanges++ & 1);
                        if (!ok) break;
                    }
                }
            } else if (row < p.n_out) {
                float* dst = p.c + static_cast<size_t>(tok0) * p.ldc + row;
#pragma unroll
                for (int i0 = 0; i0 < COLS; i0 += 16, dst += 16 * p.ldc) {
                    float old[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) old[i] = p.accumulate && tok0 + i0 + i < p.m ? dst[i * p.ldc] : 0.f;
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        if (tok0 + i0 + i < p.m) dst[i * p.ldc] = old[i] + acc[i0 + i];
                    }
                }
            }
        }
    }

    // ---- common exit: everybody (of both CTAs) meets, then the allocating warp releases tensor memory ----
    fence_before();
    __syncthreads();
    __syncwarp();
    if constexpr (PAIR) cluster_sync();
    if (warp == 1) {
        fence_after();
        if constexpr (PAIR) tmem_dealloc_pair(tmem_base, 512);
        else tmem_dealloc(tmem_base, 512);
    }
}

// [rows][k] fp16 matrix, k fastest; box = 64 elements (128 bytes) x box_rows rows, 128-byte swizzle.
int make_k_major_map(CUtensorMap* map, const void* ptr, uint64_t rows, uint64_t k, uint32_t box_rows) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return ATTN_ERR_CUDA;
    const cuuint64_t dims[2] = {k, rows};
    const cuuint64_t strides[1] = {k * 2};
    const cuuint32_t box[2] = {kStepK, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        g_last_cuda_error = static_cast<int>(r);
        return ATTN_ERR_CUDA;
    }
    return ATTN_OK;
}

struct Q8Tiling {
    bool pair;
    uint32_t parts, n_tile, t_tiles, r_tiles;
};

// The form with the least time on the busiest SM: waves of tiles x clocks per tile. Clocks of one MMA as measured for
// attn_gemm_f16 (N / 2, but no less than its shared-memory reads take: A's 128 rows 32 clocks, B's N / 4, half of them per
// CTA of a pair); a k-step is no faster than its operands arrive from L2 (~ 48 bytes per clock and SM).
Q8Tiling pick_tiling(uint32_t m, uint32_t n_out, uint32_t k, bool swiglu, uint32_t sm_count) {
    Q8Tiling best{};
    uint64_t best_cost = ~0ull;
    for (int pair = 1; pair >= 0; --pair) {
        const uint32_t workers = pair ? sm_count / 2 : sm_count;
        if (workers == 0) continue;
        for (uint32_t parts = 2; parts >= (swiglu ? 2u : 1u); --parts) {
            for (uint32_t n = 128; n >= 64; n -= 64) {
                Q8Tiling t{pair != 0, parts, n, (m + n - 1) / n, 0};
                const uint32_t span = kRowsM * (pair ? 2 : 1) * (swiglu ? 1 : parts);
                t.r_tiles = (n_out + span - 1) / span;
                const uint64_t waves = (static_cast<uint64_t>(t.t_tiles) * t.r_tiles + workers - 1) / workers;
                const uint32_t mma = std::max(n / 2, 32 + n / (pair ? 8 : 4));
                const uint64_t step = std::max<uint32_t>(8 * parts * mma, stage_bytes_of(pair != 0, parts, n) / 48);
                const uint64_t cost = waves * (k / kStepK * step + 2000 + 8 * parts * n);
                if (cost < best_cost) best_cost = cost, best = t;
            }
        }
    }
    return best;
}

bool all_aligned16(std::initializer_list<const void*> ptrs) {
    uintptr_t bits = 0;
    for (const void* q : ptrs) bits |= reinterpret_cast<uintptr_t>(q);
    return (bits & 15u) == 0;
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" int attn_gemm_q8_0(const AttnGemmQ8Args* a, void* stream_v) {
    if (!a || !a->a_hi || !a->a_lo || !a->q || !a->d || a->m == 0 || a->n_out == 0 || a->k == 0) return ATTN_ERR_INVALID_ARG;
    if (a->swiglu ? (!a->out_hi || !a->out_lo || a->accumulate) : !a->c) return ATTN_ERR_INVALID_ARG;
    if (a->k % kStepK != 0) return ATTN_ERR_UNSUPPORTED;
    const uint64_t ldc = a->ldc ? a->ldc : a->n_out;
    if (!a->swiglu && ldc < a->n_out) return ATTN_ERR_INVALID_ARG;
    if (!all_aligned16({a->a_hi, a->a_lo, a->q, a->d})) return ATTN_ERR_ALIGNMENT;
    DeviceInfo dev{};
    int rc = current_device_info(&dev);
    if (rc != ATTN_OK) return rc;
    if (dev.cc_major != 10) return ATTN_ERR_DEVICE;
    Q8GemmParams p{};
    p.c = a->c;
    p.out_hi = static_cast<__half*>(a->out_hi);
    p.out_lo = static_cast<__half*>(a->out_lo);
    p.d = static_cast<const __half*>(a->d);
    p.ldc = ldc;
    p.m = a->m;
    p.n_out = a->n_out;
    p.k = a->k;
    p.w_rows = a->n_out * (a->swiglu ? 2 : 1);
    p.d_pitch = (a->k / kBlockK + 7) & ~7u;
    p.swiglu = a->swiglu ? 1u : 0u;
    p.accumulate = a->accumulate;
    p.status = a->status;
    const Q8Tiling t = pick_tiling(p.m, p.n_out, p.k, p.swiglu != 0, static_cast<uint32_t>(dev.sm_count));
    p.t_tiles = t.t_tiles;
    p.r_tiles = t.r_tiles;
    // token tiles of a band: up to ~ 36 MB of operands, a quarter of L2, stay there while W streams past
    const uint64_t tile_bytes = static_cast<uint64_t>(t.n_tile) * p.k * 4;
    p.band = static_cast<uint32_t>(std::min<uint64_t>(t.t_tiles, std::max<uint64_t>(8, (36ull << 20) / tile_bytes)));
    const uint32_t stage_bytes = stage_bytes_of(t.pair, t.parts, t.n_tile);
    const uint32_t fixed = kTailBytes + (p.swiglu ? kExchangeBytes : 0);
    p.stages = std::min<uint32_t>(kMaxStages, (kSmemLimit - fixed) / stage_bytes);
    const uint32_t smem = p.stages * stage_bytes + fixed;
    CUtensorMap tm_w, tm_hi, tm_lo;
    if ((rc = make_k_major_map(&tm_w, a->q, p.w_rows, p.k, kRowsM)) != ATTN_OK) return rc;
    if ((rc = make_k_major_map(&tm_hi, a->a_hi, p.m, p.k, tile_tokens(t.pair, t.n_tile))) != ATTN_OK) return rc;
    if ((rc = make_k_major_map(&tm_lo, a->a_lo, p.m, p.k, tile_tokens(t.pair, t.n_tile))) != ATTN_OK) return rc;
    const uint32_t workers = static_cast<uint32_t>(dev.sm_count) / (t.pair ? 2 : 1);
    const uint32_t grid = std::min(t.t_tiles * t.r_tiles, workers) * (t.pair ? 2 : 1);
    auto pick = [&](auto pair) {
        constexpr bool P = decltype(pair)::value;
        return t.parts == 2 ? (t.n_tile == 128 ? gemm_q8_kernel<P, 2, 128> : gemm_q8_kernel<P, 2, 64>)
                            : (t.n_tile == 128 ? gemm_q8_kernel<P, 1, 128> : gemm_q8_kernel<P, 1, 64>);
    };
    auto kernel = t.pair ? pick(std::true_type{}) : pick(std::false_type{});
    B200_CUDA_TRY(allow_max_smem(kernel));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = static_cast<cudaStream_t>(stream_v);
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = t.pair ? 2 : 1;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = t.pair ? 2 : 1;
    B200_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, tm_w, tm_hi, tm_lo, p));
    g_launch_count.fetch_add(1, std::memory_order_relaxed);
    return ATTN_OK;
}

// Projection of many tokens at once (the prompt phase) on the 5th-generation tensor cores:
//
//     C[t][j] (+)= sum_i A[t][i] * W[j][i]        t < m tokens, j < n_out, i < k
//
// where the engine multiplies one token's activations by the same matrix per call (matmul() of
// include/kernels_cpu.hpp:69-80, once per prompt token from tools/infer.cpp:271-274; on the GPU the warp-per-row
// fused_gemv_clip of src/kernels.cu:117-136). W is [n_out][k] (k fastest), C is fp32.
// A arrives as two fp16 matrices, the rounded value and the rounding residual (A_hi + A_lo carries ~22 bits of the
// fp32 activation): the tensor cores multiply 16-bit operands, and one rounded operand (2^-11) would be visible in
// the greedy token stream, which has to equal the CPU path's. The engine's fp16 weights are exact: two products per
// k-step (A_hi W, A_lo W). Q8_0 weights (scale x int8, up to 18 significant bits) come as such a pair themselves
// (attn_gemm_pair): three products, A_hi W_hi, A_lo W_hi, A_hi W_lo, in ONE pass over the operands. The tensor cores
// truncate their fp32 accumulator once per k-step of 16, the largest error of the sum; with three products the
// two residual ones therefore go to an accumulator of their own and are added at the end (measured at k = 14336
// against float64: see the test), so that the large sum is truncated once per k-step and not three times.
// With `swiglu` the matrix holds gate rows followed by up rows; a tile takes equally many of each and its epilogue
// writes silu(gate) * up as the fp16 pair that the next projection reads: the fp32 gate | up matrix (1 GB at 9 000
// tokens x 28672) never exists.
//
// Kernel: persistent; a tile is 256 tokens x up to 256 outputs on a pair of CTAs (PAIR, tcgen05 cta_group::2), or
// 128 tokens on a single CTA where that pads less. Per CTA:
//   warp 0      TMA producer: A_hi, A_lo [128][64] and its share of the W tiles (half of the rows for a pair) into a
//               ring of stages, 128-byte swizzle, one mbarrier per stage (a pair's copies are all counted on the
//               leader's)
//   warp 1      one thread (of the pair's leader) issues tcgen05.mma (M 128 or 256, K 16, operands in shared memory,
//               K-major); tcgen05.commit releases the stage / hands over the accumulator in both CTAs
//   warps 2-9   epilogue: thread = token row = tensor-memory lane, two warps share a quarter of the lanes and
//               take every other 16-column chunk; a tile is read into registers at once, and its arithmetic and
//               stores overlap the next tile's MMAs
// What bounds it: the tensor pipe, and in a long prompt phase the power cap. A CTA on its own reads 64 KB of operands
// from L2 per 1024 tensor clocks; a pair shares W, and three products per load instead of 2 + 1 in two passes bring
// that to 64 KB per 1536, which is what leaves more of the power to the tensor cores.
// Tile width and pairing are chosen per shape (pick_tiling); tiles are dealt band by band of token rows whose A
// operand fits L2 next to the streamed W. Every wait is bounded.
#include <algorithm>
#include <type_traits>

#include "attn_internal.cuh"
#include "tcgen05_sm100.cuh"
#include "tma_tile.cuh"

namespace b200 {
namespace {

using namespace tc;

constexpr int GM = 128, GK = 64;
constexpr int kMaxStages = 6;
constexpr int kEpiWarps = 8;
constexpr int kGemmThreads = (2 + kEpiWarps) * 32;
constexpr uint32_t kATile = GM * GK * 2;       // 16 KB
constexpr uint32_t kHalfRowBytes = GK * 2;     // one row of a tile
constexpr uint32_t kSmemLimit = 227 * 1024;
constexpr uint32_t kTailBytes = 256 + 1024;    // barriers, tensor-memory address; slack to align the base to 1024

struct GemmParams {
    float* c;
    __half* out_hi;  // swiglu
    __half* out_lo;
    uint64_t ldc;
    uint32_t m, n_out, k;  // n_out: columns of the result (swiglu: the hidden dimension)
    uint32_t n_tile;       // MMA N, a multiple of 32 (half of it: rows of one W copy, whole 8-row groups)
    uint32_t m_tiles, n_tiles, band;
    uint32_t stages;
    uint32_t acc_cols;     // tensor-memory columns of one accumulator (128 or 256)
    uint32_t acc_bufs;     // tiles whose accumulators fit: 1 or 2
    uint32_t swiglu;
    int32_t accumulate;
    uint32_t* status;
};

constexpr uint32_t stage_bytes_of(bool pair, bool alo, bool wlo) {
    return kATile * (1 + alo) + (pair ? 1 : 2) * kATile * (1 + wlo);
}

enum { G_FULL = 0, G_EMPTY = G_FULL + kMaxStages, G_ACC_FULL = G_EMPTY + kMaxStages, G_ACC_EMPTY = G_ACC_FULL + 2,
       G_BARS = G_ACC_EMPTY + 2 };

// Tile t of the flat list: bands of `band` row tiles, inside a band the row tile varies fastest.
__device__ __forceinline__ void tile_of(const GemmParams& p, uint32_t t, uint32_t& mt, uint32_t& nt) {
    const uint32_t per_band = p.band * p.n_tiles;
    const uint32_t b = t / per_band, r = t - b * per_band;
    const uint32_t rows = min(p.band, p.m_tiles - b * p.band);
    nt = r / rows;
    mt = b * p.band + (r - nt * rows);
}

__device__ __forceinline__ void store_half_pair16(__half* hi, __half* lo, const float (&v)[16]) {
    uint32_t h[8], l[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float a = fminf(fmaxf(v[2 * i], -65504.f), 65504.f), b = fminf(fmaxf(v[2 * i + 1], -65504.f), 65504.f);
        const __half2 hh = __floats2half2_rn(a, b);
        const float2 hf = __half22float2(hh);
        const __half2 ll = __floats2half2_rn(a - hf.x, b - hf.y);
        h[i] = *reinterpret_cast<const uint32_t*>(&hh);
        l[i] = *reinterpret_cast<const uint32_t*>(&ll);
    }
    reinterpret_cast<uint4*>(hi)[0] = make_uint4(h[0], h[1], h[2], h[3]);
    reinterpret_cast<uint4*>(hi)[1] = make_uint4(h[4], h[5], h[6], h[7]);
    reinterpret_cast<uint4*>(lo)[0] = make_uint4(l[0], l[1], l[2], l[3]);
    reinterpret_cast<uint4*>(lo)[1] = make_uint4(l[4], l[5], l[6], l[7]);
}

// ALO / WLO: A / W have a residual matrix. Template arguments, so that the issuing thread's loop holds nothing but the
// wait, the MMAs and the commit.
template <bool PAIR, bool ALO, bool WLO>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_f16_kernel(const __grid_constant__ CUtensorMap tm_a_hi, const __grid_constant__ CUtensorMap tm_a_lo,
                const __grid_constant__ CUtensorMap tm_w_hi, const __grid_constant__ CUtensorMap tm_w_lo,
                const __grid_constant__ GemmParams p) {
    constexpr uint32_t kStageBytes = stage_bytes_of(PAIR, ALO, WLO);
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;  // swizzled tiles want 1024-byte alignment
    unsigned char* smem = smem_raw + (base - raw);
    const uint32_t bars_at = p.stages * kStageBytes;
    const uint32_t bars = base + bars_at;
    auto bar = [&](int i) { return bars + 8u * i; };
    volatile uint32_t* tmem_ptr_smem = reinterpret_cast<volatile uint32_t*>(smem + bars_at + G_BARS * 8);

    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const uint32_t rank = PAIR ? cluster_rank() : 0u;
    const uint32_t worker = PAIR ? blockIdx.x / 2 : blockIdx.x, workers = PAIR ? gridDim.x / 2 : gridDim.x;
    const uint32_t tiles = p.m_tiles * p.n_tiles, k_steps = p.k / GK;
    const uint32_t half_rows = p.n_tile / 2;

    if (tid == 0) {
        for (uint32_t s = 0; s < p.stages; ++s) {
            mbar_init(bar(G_FULL + s), 1);
            mbar_init(bar(G_EMPTY + s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(bar(G_ACC_FULL + a), 1);
            mbar_init(bar(G_ACC_EMPTY + a), kEpiWarps * (PAIR ? 2 : 1));  // one arrival per epilogue warp
        }
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

    if (warp == 0) {
        if (elect_one()) {
            // =============================== TMA producer ===============================
            const uint32_t half_bytes = half_rows * kHalfRowBytes;
            const uint32_t w_bytes = PAIR ? half_bytes : 2 * half_bytes;
            constexpr uint32_t w_at = (ALO ? 2 : 1) * kATile, w_pitch = (PAIR ? 1 : 2) * kATile;
            const uint32_t bytes = w_at + w_bytes * (WLO ? 2 : 1);
            uint32_t it = 0, s = 0, phase = 0;
            bool ok = true;
            for (uint32_t t = worker; t < tiles && ok; t += workers) {
                uint32_t mt, nt;
                tile_of(p, t, mt, nt);
                const int m0 = static_cast<int>(PAIR ? mt * 2 * GM + rank * GM : mt * GM);
                // the tile's two halves of W rows: consecutive, or (swiglu) gate rows and the matching up rows
                const int w0 = static_cast<int>(p.swiglu ? nt * half_rows : nt * p.n_tile);
                const int w1 = static_cast<int>(p.swiglu ? p.n_out + nt * half_rows : nt * p.n_tile + half_rows);
                for (uint32_t ks = 0; ks < k_steps; ++ks, ++it) {
                    if (it >= p.stages && !mbar_wait(bar(G_EMPTY + s), phase ^ 1)) {
                        if (p.status) atomicOr(p.status, ATTN_STATUS_WAIT_TIMEOUT);
                        ok = false;
                        break;
                    }
                    const uint32_t dst = base + s * kStageBytes;
                    const uint32_t full = bar(G_FULL + s);
                    const int kc = static_cast<int>(ks * GK);
                    auto load = [&](uint32_t at, const CUtensorMap* map, int row) {
                        if constexpr (PAIR) tma_load_2d_pair(dst + at, map, full, kc, row);
                        else tma_load_2d(dst + at, map, full, kc, row);
                    };
                    if (rank == 0) mbar_arrive_expect_tx(full, PAIR ? 2 * bytes : bytes);
                    load(0, &tm_a_hi, m0);
                    if constexpr (ALO) load(kATile, &tm_a_lo, m0);
                    if constexpr (PAIR) {
                        load(w_at, &tm_w_hi, rank ? w1 : w0);
                        if constexpr (WLO) load(w_at + w_pitch, &tm_w_lo, rank ? w1 : w0);
                    } else {
                        load(w_at, &tm_w_hi, w0);
                        load(w_at + half_bytes, &tm_w_hi, w1);
                        if constexpr (WLO) {
                            load(w_at + w_pitch, &tm_w_lo, w0);
                            load(w_at + w_pitch + half_bytes, &tm_w_lo, w1);
                        }
                    }
                    if (++s == p.stages) s = 0, phase ^= 1;
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && elect_one()) {
            // =============================== MMA issuer ===============================
            const uint32_t idesc = instr_desc(0, 0, 0, PAIR ? 2 * GM : GM, p.n_tile);
            constexpr uint32_t w_at = (ALO ? 2 : 1) * kATile, w_pitch = (PAIR ? 1 : 2) * kATile;
            auto mma = [&](uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
                if constexpr (PAIR) mma_ss_pair(d, a, b, idesc, acc);
                else mma_ss(d, a, b, idesc, acc);
            };
            auto done = [&](uint32_t b) {
                if constexpr (PAIR) commit_pair(b);
                else commit(b);
            };
            const uint64_t desc0 = smem_desc(base, 16, 1024);
            uint32_t local = 0, s = 0, phase = 0;
            bool ok = true;
            for (uint32_t t = worker; t < tiles && ok; t += workers, ++local) {
                const uint32_t a = p.acc_bufs == 2 ? local & 1 : 0;
                if (local >= p.acc_bufs && !mbar_wait(bar(G_ACC_EMPTY + a), (local / p.acc_bufs - 1) & 1)) {
                    if (p.status) atomicOr(p.status, ATTN_STATUS_WAIT_TIMEOUT);
                    break;
                }
                fence_after();
                const uint32_t d = tmem_base + a * 256;  // (two buffers: 256 columns apart either way)
                // residual products: into their own accumulator when W has a residual too
                const uint32_t d_lo = WLO ? d + p.acc_cols : d;
                for (uint32_t ks = 0; ks < k_steps; ++ks) {
                    if (!mbar_wait(bar(G_FULL + s), phase)) {
                        if (p.status) atomicOr(p.status, ATTN_STATUS_WAIT_TIMEOUT);
                        ok = false;
                        break;
                    }
                    fence_after();
                    // K-major operands, 128-byte swizzle: 32 bytes per k-step of 16, 8-row groups 1024 bytes apart
                    const uint64_t a_hi = desc0 + s * (kStageBytes / 16), a_lo = a_hi + kATile / 16;  // (in 16 bytes)
                    const uint64_t w_hi = a_hi + w_at / 16, w_lo = w_hi + w_pitch / 16;
#pragma unroll
                    for (int kk = 0; kk < GK / 16; ++kk) {
                        const uint32_t more = (ks | kk) != 0;
                        mma(d, a_hi + 2 * kk, w_hi + 2 * kk, more);
                        if constexpr (ALO) mma(d_lo, a_lo + 2 * kk, w_hi + 2 * kk, WLO ? more : 1u);
                        if constexpr (WLO) mma(d_lo, a_hi + 2 * kk, w_lo + 2 * kk, ALO ? 1u : more);
                    }
                    done(bar(G_EMPTY + s));  // the stage may be refilled once these MMAs have read it
                    if (++s == p.stages) s = 0, phase ^= 1;
                }
                if (ok) done(bar(G_ACC_FULL + a));
            }
        }
    } else {
        // =============================== epilogue warps ===============================
        const uint32_t quarter = warp & 3;                      // the tensor-memory lanes this warp may read
        const uint32_t first = (warp - 2) >> 2;                 // even or odd 16-column chunks
        const uint32_t lane_addr = (quarter * 32) << 16;
        const uint32_t chunks = (p.swiglu ? half_rows : p.n_tile) / 16;
        uint32_t local = 0;
        for (uint32_t t = worker; t < tiles; t += workers, ++local) {
            const uint32_t a = p.acc_bufs == 2 ? local & 1 : 0;
            uint32_t mt, nt;
            tile_of(p, t, mt, nt);
            const uint32_t row = (PAIR ? mt * 2 * GM + rank * GM : mt * GM) + quarter * 32 + lane;
            const uint32_t n0 = nt * (p.swiglu ? half_rows : p.n_tile);
            const bool live = row < p.m;
            // The vote brings the warp together again (lanes past m leave a tile early, and tcgen05.ld wants the whole warp)
            // and lets all its lanes give up or go on.
            if (!__all_sync(0xffffffffu, mbar_wait(bar(G_ACC_FULL + a), (local / p.acc_bufs) & 1))) {
                if (lane == 0 && p.status) atomicOr(p.status, ATTN_STATUS_WAIT_TIMEOUT);
                break;
            }
            fence_after();
            // Everything this thread owns of the tile goes to registers first (up to eight chunks of 16 columns; swiglu:
            // four of the gate, four of the up half), so that the accumulator is free for the next tile's MMAs before
            // the arithmetic and the stores begin.
            const uint32_t acc = tmem_base + a * 256 + lane_addr;
            float v[8][16];
            auto load = [&](uint32_t at) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint32_t c = p.swiglu ? first + 2 * (j & 3) : first + 2 * j;
                    if (c < chunks) tmem_ld16(at + c * 16 + (p.swiglu && j >= 4 ? half_rows : 0), v[j]);
                }
                tmem_wait_ld();
            };
            load(acc);
            if constexpr (WLO) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint32_t c = p.swiglu ? first + 2 * (j & 3) : first + 2 * j;
                    if (c < chunks) {
                        float lo[16];
                        tmem_ld16(acc + p.acc_cols + c * 16 + (p.swiglu && j >= 4 ? half_rows : 0), lo);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 16; ++i) v[j][i] += lo[i];
                    }
                }
            }
            fence_before();
            __syncwarp();
            if (lane == 0) {
                if constexpr (PAIR) mbar_arrive_cluster(bar(G_ACC_EMPTY + a), 0);
                else mbar_arrive(bar(G_ACC_EMPTY + a));
            }
            if (!live) continue;
            if (p.swiglu) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t c = first + 2 * j;
                    if (c < chunks && n0 + c * 16 < p.n_out) {   // n_out is a multiple of 16
                        // silu(x) = x / (1 + expf(-x)), src/model/block.cpp:206-210
#pragma unroll
                        for (int i = 0; i < 16; ++i) v[j][i] = __fdiv_rn(v[j][i], 1.0f + expf(-v[j][i])) * v[j + 4][i];
                        const size_t o = static_cast<size_t>(row) * p.n_out + n0 + c * 16;
                        store_half_pair16(p.out_hi + o, p.out_lo + o, v[j]);
                    }
                }
            } else {
                float4* crow = reinterpret_cast<float4*>(p.c + static_cast<size_t>(row) * p.ldc + n0);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint32_t c = first + 2 * j;
                    if (c < chunks && n0 + c * 16 < p.n_out) {
                        float4* dst = crow + c * 4;
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            float4 o = make_float4(v[j][4 * i], v[j][4 * i + 1], v[j][4 * i + 2], v[j][4 * i + 3]);
                            if (p.accumulate) {
                                const float4 old = dst[i];
                                o.x += old.x, o.y += old.y, o.z += old.z, o.w += old.w;
                            }
                            dst[i] = o;
                        }
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
    const cuuint32_t box[2] = {GK, box_rows};
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

struct Tiling {
    bool pair;
    uint32_t n_tile, m_tiles, n_tiles;
};

// Pairing and tile width with the least time on the busiest SM: waves of tiles x clocks per tile. Clocks of one MMA,
// measured with the operands in place: N / 2 (the tensor pipe; a pair's covers twice the rows in the same time), but no
// less than its shared-memory reads take (A's 128 rows 32 clocks, B's N rows N / 4, half of them per CTA of a pair:
// N = 128 measured 64.3 clocks, N = 64 48.2); a k-step is no faster than its operands arrive from L2 (~ 48 bytes per
// clock and SM). 1003 tokens x 28672 on 74 pairs: width 256 makes 448 tiles = 7 waves of 256, width 224 512 tiles =
// 7 waves of 224.
Tiling pick_tiling(uint32_t m, uint32_t n_out, uint32_t k, bool swiglu, bool has_alo, bool has_wlo, uint32_t sm_count) {
    Tiling best{};
    uint64_t best_cost = ~0ull;
    const uint32_t products = 1 + has_alo + has_wlo;
    for (int pair = 1; pair >= 0; --pair) {
        const uint32_t rows = pair ? 2 * GM : GM, workers = pair ? sm_count / 2 : sm_count;
        if (workers == 0 || (pair && m <= GM)) continue;
        for (uint32_t n = 256; n >= (pair ? 64u : 32u); n -= 32) {
            Tiling t{pair != 0, n, (m + rows - 1) / rows, 0};
            const uint32_t width = swiglu ? n / 2 : n;
            t.n_tiles = (n_out + width - 1) / width;
            const uint64_t waves = (static_cast<uint64_t>(t.m_tiles) * t.n_tiles + workers - 1) / workers;
            const uint32_t mma = std::max(n / 2, 32 + n / (pair ? 8 : 4));
            const uint32_t bytes = kATile * (1 + has_alo) + n * kHalfRowBytes / (pair ? 2 : 1) * (1 + has_wlo);
            const uint64_t step = std::max<uint32_t>(products * (GK / 16) * mma, bytes / 48);
            // what a tile costs besides: its first operands and, with one accumulator, its epilogue
            const uint64_t cost = waves * (k / GK * step + (has_wlo ? 3000 + 8 * n : 1000));
            if (cost < best_cost) best_cost = cost, best = t;
        }
    }
    return best;
}

int launch_gemm(GemmParams& p, const void* a_hi, const void* a_lo, const void* w_hi, const void* w_lo, void* stream_v) {
    DeviceInfo dev{};
    int rc = current_device_info(&dev);
    if (rc != ATTN_OK) return rc;
    if (dev.cc_major != 10) return ATTN_ERR_DEVICE;
    const Tiling t = pick_tiling(p.m, p.n_out, p.k, p.swiglu != 0, a_lo != nullptr, w_lo != nullptr,
                                 static_cast<uint32_t>(dev.sm_count));
    const bool alo = a_lo != nullptr, wlo = w_lo != nullptr;
    p.n_tile = t.n_tile;
    p.m_tiles = t.m_tiles;
    p.n_tiles = t.n_tiles;
    // rows of A of a band: up to ~ 36 MB of operands, a quarter of L2, stay there while W streams past, but at least four
    // row tiles, so that a W tile is used that often (k = 14336, a pair, value and residual: 59 MB)
    const uint64_t row_tile_bytes = static_cast<uint64_t>(t.pair ? 2 : 1) * GM * p.k * 2 * (1 + alo);
    p.band = static_cast<uint32_t>(std::min<uint64_t>(t.m_tiles, std::max<uint64_t>(4, (36ull << 20) / row_tile_bytes)));
    p.acc_cols = t.n_tile <= 128 ? 128 : 256;
    p.acc_bufs = wlo && p.acc_cols == 256 ? 1 : 2;
    const uint32_t stage_bytes = stage_bytes_of(t.pair, alo, wlo);
    p.stages = std::min<uint32_t>(kMaxStages, (kSmemLimit - kTailBytes) / stage_bytes);
    const uint32_t smem = p.stages * stage_bytes + kTailBytes;
    CUtensorMap tm_ahi, tm_alo, tm_whi, tm_wlo;
    const uint64_t w_rows = static_cast<uint64_t>(p.n_out) * (p.swiglu ? 2 : 1);
    if ((rc = make_k_major_map(&tm_ahi, a_hi, p.m, p.k, GM)) != ATTN_OK) return rc;
    if ((rc = make_k_major_map(&tm_alo, a_lo ? a_lo : a_hi, p.m, p.k, GM)) != ATTN_OK) return rc;
    if ((rc = make_k_major_map(&tm_whi, w_hi, w_rows, p.k, t.n_tile / 2)) != ATTN_OK) return rc;
    if ((rc = make_k_major_map(&tm_wlo, w_lo ? w_lo : w_hi, w_rows, p.k, t.n_tile / 2)) != ATTN_OK) return rc;
    const uint32_t workers = static_cast<uint32_t>(dev.sm_count) / (t.pair ? 2 : 1);
    const uint32_t grid = std::min(t.m_tiles * t.n_tiles, workers) * (t.pair ? 2 : 1);
    auto pick = [&](auto pair) {
        constexpr bool P = decltype(pair)::value;
        return alo ? (wlo ? gemm_f16_kernel<P, true, true> : gemm_f16_kernel<P, true, false>)
                   : (wlo ? gemm_f16_kernel<P, false, true> : gemm_f16_kernel<P, false, false>);
    };
    auto kernel = t.pair ? pick(std::true_type{}) : pick(std::false_type{});
    B200_CUDA_TRY(allow_max_smem(kernel));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kGemmThreads);
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
    B200_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, tm_ahi, tm_alo, tm_whi, tm_wlo, p));
    g_launch_count.fetch_add(1, std::memory_order_relaxed);
    return ATTN_OK;
}

bool all_aligned16(std::initializer_list<const void*> ptrs) {
    uintptr_t bits = 0;
    for (const void* q : ptrs) bits |= reinterpret_cast<uintptr_t>(q);
    return (bits & 15u) == 0;
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" int attn_gemm_f16(const AttnGemmArgs* a, void* stream_v) {
    if (!a || !a->c || !a->a_hi || !a->w || a->m == 0 || a->n_out == 0 || a->k == 0) return ATTN_ERR_INVALID_ARG;
    if (a->k % GK != 0 || a->n_out % 32 != 0) return ATTN_ERR_UNSUPPORTED;
    const uint64_t ldc = a->ldc ? a->ldc : a->n_out;
    if (ldc < a->n_out || ldc % 4 != 0) return ATTN_ERR_INVALID_ARG;
    if (!all_aligned16({a->c, a->a_hi, a->a_lo, a->w})) return ATTN_ERR_ALIGNMENT;
    GemmParams p{};
    p.c = a->c;
    p.ldc = ldc;
    p.m = a->m;
    p.n_out = a->n_out;
    p.k = a->k;
    p.accumulate = a->accumulate;
    p.status = a->status;
    return launch_gemm(p, a->a_hi, a->a_lo, a->w, nullptr, stream_v);
}

extern "C" int attn_gemm_pair(const AttnGemmPairArgs* a, void* stream_v) {
    if (!a || !a->a_hi || !a->w_hi || a->m == 0 || a->n_out == 0 || a->k == 0) return ATTN_ERR_INVALID_ARG;
    if (a->swiglu ? (!a->out_hi || !a->out_lo || a->accumulate) : !a->c) return ATTN_ERR_INVALID_ARG;
    if (a->k % GK != 0 || a->n_out % 32 != 0) return ATTN_ERR_UNSUPPORTED;
    const uint64_t ldc = a->ldc ? a->ldc : a->n_out;
    if (!a->swiglu && (ldc < a->n_out || ldc % 4 != 0)) return ATTN_ERR_INVALID_ARG;
    if (!all_aligned16({a->c, a->a_hi, a->a_lo, a->w_hi, a->w_lo, a->out_hi, a->out_lo})) return ATTN_ERR_ALIGNMENT;
    GemmParams p{};
    p.c = a->c;
    p.out_hi = static_cast<__half*>(a->out_hi);
    p.out_lo = static_cast<__half*>(a->out_lo);
    p.ldc = ldc;
    p.m = a->m;
    p.n_out = a->n_out;
    p.k = a->k;
    p.swiglu = a->swiglu ? 1u : 0u;
    p.accumulate = a->accumulate;
    p.status = a->status;
    return launch_gemm(p, a->a_hi, a->a_lo, a->w_hi, a->w_lo, stream_v);
}

// Decode attention in ONE launch for short and middling contexts: a cluster of CTAs per segment (sequence x kv-head group),
// which merges its own partials over distributed shared memory (kernel body: decode_body.cuh, CLUSTER).
//
// The two-launch form deals all tiles evenly over the SMs and merges in a second kernel; that kernel, the partials' way through
// L2 and the dependency between the two cost 3 to 5 us of device time and a launch, whatever the length. Here a segment's
// share of the SMs is fixed, so ragged lengths leave SMs idle; that is the price, and an estimate of both decides
// (pick_decode_cluster). What bounds it: up to a few tiles per CTA the chain launch - query - first tile - merge (5 us), then
// one SM's rate over its own tiles (0.74 us per 64 KB) or the HBM: 16 x 4096 rows of 8 heads of 128 44.0 us (6.1 TB/s, 47.3 in
// the two-launch form), 8 x 2048 14.7 (17.6), 1 x 4096 9.7 (10.8), 16 x up to 1000 of 4 heads of 64 7.8 (12.3).
#include <algorithm>
#include <atomic>

#include "decode_body.cuh"
#include "tma_tile.cuh"

namespace b200 {

namespace {

using decode_detail::kConsumerWarps;
using decode_detail::kThreads;

constexpr uint32_t kMaxCluster = 8;  // portable

// Bytes per ns: one SM over its own tiles (0.74 us per 64 KB tile), and the HBM.
constexpr double kSmRate = 88, kHbmRate = 6500;
// What the cluster form saves besides its streaming time with one length for all, measured as the difference of the two forms'
// times in graphs of calls beyond their streaming: 2.8 us (8 x 2048 rows 17.6 -> 14.7 us, 1 x 4096 10.7 -> 9.6), less a margin (1 x
// 8192 rows: 12.8 split, 13.1 in clusters). kCtaNs: one more CTA in a cluster's barriers and merge (time stamps from the last tile to
// the last store: 2.3 us with one CTA per cluster, 3.9 with eight, twice this value at most; it decides between plans whose
// tiles take the same time).
constexpr double kGainNs = 1500, kCtaNs = 100;

// Ragged lengths are on the device; the host knows how long the caches are, not how they are filled. A segment's share of the
// SMs is fixed here, so a long sequence among short ones is the worst that can happen (16 caches of 4096 rows, one of them
// full: 32.6 us, split pass 22.0; all full: 44.0 and 49.4), and the rule looks at that: clusters only where they lose to the
// split pass for no number of full caches. Both estimates without what each form always takes (kRaggedGainNs apart):
//   clusters     the longest sequence's tiles on its own SMs (kTileNs each, under load)
//   split pass   its tiles dealt over all SMs, a bulk copy per row and cache (kCopyNs + kCopyKbNs per KB), the HBM, and where
//                a warp merges a row by itself (kMergeWarpRows) the partials of a row one after the other
// Checked on 660 shapes (1 to 48 caches of 256 to 16384 rows, five head geometries, 1 to all of them full, the others 100
// rows): of the ~ 350 that take the clusters one loses, by 3 % (1 x 8192 with 64 heads), and all fillings together run 1.6 times as
// fast as in the split form. The rule before, which took every batch as 56 % full, took 550 and lost in 191, by up to 7 times.
constexpr double kTileNs128 = 840, kTileNs64 = 580, kRaggedGainNs = 1850;
constexpr double kCopyNs = 30, kCopyKbNs = 12, kPartialNs = 60;

// The split form with `full` caches of `rows` rows and the others next to empty.
double split_ns(const DecodePlan& s, uint32_t rows, uint32_t full, uint32_t merge_rows, uint32_t min_tiles, uint32_t head_dim) {
    const uint64_t tiles = static_cast<uint64_t>(full) * s.head_groups * ((rows + s.tile_rows - 1) / s.tile_rows);
    const uint32_t ctas = active_ctas(s.grid, 0, min_tiles, tiles);
    const uint32_t row_bytes = s.hpc * head_dim * 2;
    const double copies = static_cast<double>((tiles + ctas - 1) / ctas) * 2 * s.tile_rows * (kCopyNs + kCopyKbNs / 1024 * row_bytes);
    const double streaming = 2.0 * full * rows * s.head_groups * row_bytes / kHbmRate;
    const double merge = merge_rows >= kMergeWarpRows ? kPartialNs * ctas / (full * s.head_groups) : 0;
    return std::max(copies, streaming) + merge;
}

template <int D, int HPC, bool QSPLIT, bool BF16>
__global__ void __launch_bounds__(kThreads, 1) decode_cluster_kernel(const __grid_constant__ DecodeParams p,
                                                                     const __grid_constant__ CUtensorMap tm_k,
                                                                     const __grid_constant__ CUtensorMap tm_v) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);  // swizzled tiles want 1024-byte alignment
    decode_detail::decode_split_body<D, HPC, QSPLIT, BF16, /*FUSED=*/false, /*LOW8=*/false, /*PACK8=*/true, /*CLUSTER=*/true>(
        p, smem, &tm_k, &tm_v);
}

using Kernel = void (*)(DecodeParams, CUtensorMap, CUtensorMap);

template <int D, bool QSPLIT, bool BF16>
Kernel kernel_hpc(uint32_t hpc) {
    switch (hpc) {
        case 8: return decode_cluster_kernel<D, 8, QSPLIT, BF16>;
        case 4: return decode_cluster_kernel<D, 4, QSPLIT, BF16>;
        case 2: return decode_cluster_kernel<D, 2, QSPLIT, BF16>;
        default: return decode_cluster_kernel<D, 1, QSPLIT, BF16>;
    }
}
template <int D>
Kernel kernel_types(uint32_t hpc, bool qsplit, bool kv_bf16) {
    if (kv_bf16) return kernel_hpc<D, true, true>(hpc);
    return qsplit ? kernel_hpc<D, true, false>(hpc) : kernel_hpc<D, false, false>(hpc);
}
Kernel kernel_of(uint32_t head_dim, uint32_t hpc, bool qsplit, bool kv_bf16) {
    return head_dim == 128 ? kernel_types<128>(hpc, qsplit, kv_bf16) : kernel_types<64>(hpc, qsplit, kv_bf16);
}

void launch_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&attr)[2], uint32_t grid, uint32_t cluster, size_t smem,
                   cudaStream_t stream) {
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
}

// Clusters of this size that run at once with one CTA per SM (how the SMs are grouped differs between GPUs): asked once per
// device and size, of one kernel for all, because every form takes more than half of an SM's shared memory.
uint32_t resident_clusters(uint32_t cluster, const DeviceInfo& dev) {
    constexpr int kMaxDevices = 64;
    static std::atomic<int> cache[kMaxDevices][kMaxCluster];  // 0 = not asked yet, else the count + 1
    if (dev.device < 0 || dev.device >= kMaxDevices) return 0;
    std::atomic<int>& slot = cache[dev.device][cluster - 1];
    int known = slot.load(std::memory_order_acquire);
    if (known == 0) {
        const size_t smem = static_cast<size_t>(dev.max_smem_optin);
        const Kernel kernel = kernel_of(128, 8, true, false);
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute attr[2];
        launch_config(cfg, attr, cluster, cluster, smem, nullptr);
        cfg.numAttrs = 1;
        int n = 0;
        if (allow_max_smem(kernel) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
            (void)cudaGetLastError();
            n = 0;
        }
        known = n + 1;
        slot.store(known, std::memory_order_release);
    }
    return static_cast<uint32_t>(known - 1);
}

// K or V caches as [sequence][kv head][128-byte part of a head][row][64 elements]; box = all parts of hpc heads over a tile's
// rows. Rows past `rows` read as zeros.
bool cache_map(CUtensorMap* map, const void* cache, const DecodeParams& p, uint32_t head_dim, uint32_t rows, uint32_t hpc,
               bool bf16) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return false;
    const uint64_t row_bytes = p.kv_row_stride * 2, batch_bytes = p.batch > 1 ? p.kv_batch_stride * 2 : row_bytes * rows;
    const cuuint64_t dims[5] = {64, rows, head_dim / 64, p.n_kv_heads, p.batch};
    const cuuint64_t strides[4] = {row_bytes, 128, static_cast<cuuint64_t>(head_dim) * 2, batch_bytes};
    const cuuint32_t box[5] = {64, 16u * (kConsumerWarps / hpc), head_dim / 64, hpc, 1};
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    return enc(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5, const_cast<void*>(cache), dims,
               strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

bool pick_decode_cluster(uint32_t batch, uint32_t n_heads, uint32_t n_kv_heads, uint32_t head_dim, uint32_t rows, bool ragged,
                         const DecodePlan& split, uint32_t split_min_tiles, const DeviceInfo& dev, DecodeClusterPlan* plan) {
    if (rows == 0 || n_heads / n_kv_heads > 8) return false;
    const double one = 4.0 * rows * n_kv_heads * head_dim / kHbmRate;  // streaming of one full cache
    const double streaming = ragged ? one : batch * one;
    double best = 1e30;
    uint32_t best_hpc = 0, best_cluster = 0;
    for (uint32_t hpc = 8; hpc >= 1; hpc /= 2) {
        if (n_kv_heads % hpc != 0) continue;
        const uint64_t segments = static_cast<uint64_t>(batch) * (n_kv_heads / hpc);
        const uint32_t tile_rows = 16 * (kConsumerWarps / hpc), tiles = (rows + tile_rows - 1) / tile_rows;
        const double tile_ns = !ragged ? 4.0 * tile_rows * hpc * head_dim / kSmRate : head_dim == 128 ? kTileNs128 : kTileNs64;
        for (uint32_t c = kMaxCluster; c >= 1; --c) {
            if (segments > resident_clusters(c, dev)) continue;  // (all of them at once: a second round would double the time)
            const double t = std::max(((tiles + c - 1) / c) * tile_ns, streaming) + kCtaNs * c;
            if (t < best) best = t, best_hpc = hpc, best_cluster = c;
        }
    }
    if (best_hpc == 0) return false;
    if (!ragged) {
        if (best > streaming + kGainNs) return false;
    } else {
        for (uint32_t full = 1;; full = std::min(2 * full, batch)) {
            const double split_time = split_ns(split, rows, full, batch * n_heads, split_min_tiles, head_dim);
            if (std::max(best, full * one) > split_time + kRaggedGainNs) return false;
            if (full == batch) break;
        }
    }
    // ring of K and V tiles, then as in the split pass: query rows of one segment, barriers, two words behind a prefix that
    // this form does not use; the base is aligned to 1024
    const size_t tile = static_cast<size_t>(16 * (kConsumerWarps / best_hpc)) * best_hpc * head_dim * 2;
    const uint32_t segments = batch * (n_kv_heads / best_hpc);
    const size_t fixed = 1024 + 16 + static_cast<size_t>(best_hpc) * (n_heads / n_kv_heads) * head_dim * 4 +
                         (static_cast<size_t>(segments) + 1) * 4 + 128;
    const size_t stages = std::min<size_t>(8, (static_cast<size_t>(dev.max_smem_optin) - fixed) / (2 * tile + 24));
    if (stages < 2) return false;
    plan->rows = rows;
    plan->hpc = best_hpc;
    plan->cluster = best_cluster;
    plan->stages = static_cast<uint32_t>(stages);
    plan->segments = segments;
    plan->smem_bytes = stages * (2 * tile + 24) + fixed;
    return true;
}

int launch_decode_cluster(const DecodeParams& p, const DecodeClusterPlan& plan, uint32_t head_dim, bool qsplit, bool kv_bf16,
                          cudaStream_t stream) {
    CUtensorMap tm_k, tm_v;
    if (!cache_map(&tm_k, p.k, p, head_dim, plan.rows, plan.hpc, kv_bf16) ||
        !cache_map(&tm_v, p.v, p, head_dim, plan.rows, plan.hpc, kv_bf16))
        return kClusterNotTaken;  // (strides beyond what a tensor map holds)
    const Kernel kernel = kernel_of(head_dim, plan.hpc, qsplit, kv_bf16);
    B200_CUDA_TRY(allow_max_smem(kernel));
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[2];
    launch_config(cfg, attr, plan.segments * plan.cluster, plan.cluster, plan.smem_bytes, stream);
    B200_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, p, tm_k, tm_v));
    g_launch_count.fetch_add(1, std::memory_order_relaxed);
    return ATTN_OK;
}

}  // namespace b200

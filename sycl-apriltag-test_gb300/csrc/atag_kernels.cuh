// atag_kernels.cuh — per-frame device descriptors and kernel declarations.
#pragma once

#include "atag_device.cuh"

namespace atag {

// Everything a kernel needs to know about one frame: its size and where its
// buffers live in the workspace.  A batch is an array of these in device
// memory; kernels pick their frame from blockIdx.y (pixel stages),
// blockIdx.x (boundary points) or a flattened work index (cluster stages).
struct FrameDesc {
    // sizes
    uint32_t width, height;            // after decimation
    uint32_t factor;                   // decimation factor
    uint32_t src_stride;               // source row pitch in bytes
    uint32_t src_format;               // atag_pixel_format of the source
    // pixel buffers
    const uint8_t* src;                // source frame (before decimation)
    uint8_t* grey;                     // decimated grey frame (== src when grey and factor 1)
    uint8_t* thr;                      // thresholded
    uint8_t* extrema;                  // optional tile min/max (2 B / tile)
    uint8_t* filtered_extrema;         // optional dilated min/max
    uint32_t* scratch;                 // union-find forest (w*h)
    uint32_t* labels;                  // w*h
    uint32_t* sizes;                   // w*h
    atag_boundary_point* dense_points; // optional 4 planes (drop-in find_boundaries)
    uint64_t* dense_keys;              // optional 4 planes
    // boundary points grouped by pair (fused path)
    unsigned long long* points;        // (pair slot << 32) | packed point
    uint32_t point_cap;
    // pair hash table
    uint32_t pair_cap;                 // power of two
    unsigned long long* pair_keys;     // EMPTY = ~0
    uint4* pair_bbox;                  // x_min, x_max, y_min, y_max (2x coords)
    int2* pair_gsum;                   // gx_sum, gy_sum
    unsigned long long* pair_pxgx;     // pxgx_pygy_sum
    uint32_t* pair_count;
    uint32_t* pair_cluster;            // slot -> filtered cluster index or INVALID
    // filtered clusters (sorted by pair key)
    uint32_t cluster_cap;
    unsigned long long* cluster_keys;
    atag_cluster_bounds* cluster_bounds;
    atag_cluster_extents* cluster_extents;
    float2* cluster_center;            // (cx, cy)
    uint32_t* cluster_cursor;
    uint32_t* peak_count;              // per cluster
    atag_corner* peaks;                // per cluster x 10
    uint32_t* peak_clusters;           // rank q -> cluster
    atag_peak_extents* peak_extents;   // rank q -> {start, count}
    atag_fitted_quad* fitted;          // per rank q
    atag_quad_corners* quad_tmp;       // per rank q
    uint32_t* quad_ok;                 // per rank q
    // cluster points
    uint32_t cpoint_cap;
    unsigned long long* sortbuf;       // (theta key << 32) | packed; then the sorted points' line-fit inputs
    atag_cluster_point* cluster_points;
    atag_line_fit_point* line_fit;
    float* errbuf;                     // 8 bytes per point: sort scratch of clusters past the shared memory,
                                       // then the corner candidates
    uint32_t* cluster_work;            // small clusters from the front, large from the back
    uint32_t* cluster_runs;            // first run (CE_RUN points) of each cluster
    struct RunInfo* runs;              // per run
    // outputs
    atag_quad_corners* quads;
    uint32_t quad_cap;
    atag_frame_stats* stats;
    uint32_t* counters;                // per-frame work counters (see Counter)
    // DEAD_PAIRS label word pairs (white << 32 | black, EMPTY = ~0) of pairs
    // whose running point count is already above the cluster size limit; null
    // when not tracked
    unsigned long long* dead_pairs;
    // iteration cap of the frame-wide union-find loops (0: the default that the
    // tile count gives, see k_pixels.cu)
    uint32_t uf_cap;
    // optional (stage entry point): every pair's ClusterBounds and key in
    // key order, up to pair_out_cap entries; null in the fused path
    atag_cluster_bounds* pair_bounds_out;
    unsigned long long* pair_keys_out;
    uint32_t pair_out_cap;
    // 1: write the reference's complete segmentation arrays (every parent
    // compressed to its root, block information words at odd rows, zero
    // sizes away from roots).  0 (fused batches): only what later stages
    // read, i.e. parents at even rows and sizes at the roots.
    uint32_t stage_outputs;
    // Tile CCL edge records (ccl_edge_words(tile rows) words per CCL tile,
    // see k_pixels.cu): the tile roots and cross-tile links of each tile's
    // edge blocks, written by the tile pass and read by the border pass.
    // Null: the border pass reads the thresholded image and the forest.
    uint32_t* edges;
};

// Words of one CCL tile's edge record (tiles of 32 blocks x `rows` block
// rows): per edge block a (255 slot, 0 slot) pair of tile roots whose bits
// 24-27 hold that forest's P, Q, R, S links: the top row [0, 32), the
// bottom row [32, 64), the left column [64, 64 + rows), the right column
// [64 + rows, 64 + 2 rows).
__host__ __device__ constexpr uint32_t ccl_edge_words(uint32_t rows) { return 2 * (64 + 2 * rows); }

// The frames a launch works on: a device table (batches) or one descriptor
// passed by value (stage entry points, which must not allocate).  Kernels
// receive it as a __grid_constant__ parameter, so `one` is read in place.
struct FrameSet {
    const FrameDesc* table;
    FrameDesc one;
    uint32_t overlap;  // launched to overlap the previous kernel's end (await_previous_kernel)
    __device__ __forceinline__ const FrameDesc& get(uint32_t i) const { return table ? table[i] : one; }
    // In kernels of the detector's path only.  Fields behind the choice above are
    // read by generic loads; by global ones the boundary pass of 64 1080p frames
    // took 870 instead of 890 us and their tile labelling 654 instead of 664.
    __device__ __forceinline__ const FrameDesc& of_table(uint32_t i) const { return table[i]; }
};

// First in every kernel of the detector's path when it is launched with
// fs.overlap: its CTAs may then be placed on the SMs while the kernel before
// it still runs (programmatic dependent launch).  The first call returns when
// that kernel, and with it everything before it, has finished; the second lets
// the next kernel's CTAs be placed once all of this kernel's have started.
// The compiler may move a read-only load (__ldg, const __restrict__) up across
// the wait, so one of data that an earlier kernel wrote goes through a
// descriptor's pointer that is itself read, by a plain load, after it.
// Large lanes beside others run without (launch_lane), and so do captures: the
// calls alone made their pixel kernels, of up to half a million short CTAs, 1-4%
// slower, so those are compiled both ways.
__device__ __forceinline__ void await_previous_kernel() {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
}

// per-frame counters (FrameDesc::counters[...])
enum Counter : uint32_t {
    CNT_POINTS = 0,      // boundary points written
    CNT_STATUS = 1,      // ATAG_DEVFLAG_* bits
    CNT_CLUSTERS = 2,    // filtered clusters
    CNT_PEAKCLU = 3,     // clusters with peaks
    CNT_WORK = 4,        // work-queue cursor
    CNT_ALLPOINTS = 5,   // boundary points found (list entries of pairs already
                         // known to exceed the cluster size limit are skipped)
    CNT_SMALL = 6,       // clusters of at most CF_SMALL_CAP points
    CNT_LARGE = 7,       // larger clusters
    CNT_RUNS = 8,        // runs of up to CE_RUN points of one cluster
    CNT_PAIRS = 9,       // distinct pairs (entries of the frame's key list)
    CNT_COUNT = 10
};

constexpr uint32_t DEAD_PAIRS = 2;

// Cluster-sort kernel shapes: most clusters are small and run several per SM
// on 256 threads, large ones get a 1024-thread CTA.  Keys sort in shared
// memory: a large CTA's is sized for the largest cluster that passes the
// filter (2 (2 w + 2 h) points, cluster_bounds.h:92-93), up to CF_LARGE_CAP
// (every frame up to 3840 x 2160).
constexpr uint32_t CF_SMALL_THREADS = 256, CF_SMALL_CAP = 2048, CF_SMALL_NB = 2048;
constexpr uint32_t CF_LARGE_THREADS = 1024, CF_LARGE_CAP = 24576, CF_LARGE_NB = 4096;
__host__ __device__ constexpr uint32_t cf_smem(uint32_t cap, uint32_t nb) { return cap * 8 + nb * 4; }
constexpr uint32_t CF_LARGE_SMEM = cf_smem(CF_LARGE_CAP, CF_LARGE_NB);
__host__ __device__ constexpr uint32_t max_cluster_points(uint32_t w, uint32_t h) { return 2 * (2 * w + 2 * h); }
// A run: up to CE_RUN consecutive points of one cluster, the work item of a
// warp in the prefix-sum and window-error kernels.
constexpr uint32_t CE_RUN = 256;
constexpr uint32_t CF_MAX_RUNS = max_cluster_points(4096, 4096) / CE_RUN;
struct RunInfo {
    long long before[6];  // moments (Mx, My, Mxx, Myy, Mxy, W) of the cluster's earlier runs
    uint32_t cluster, first;  // its cluster and first point in it
    uint32_t pad_[2];
};
__host__ __device__ constexpr size_t max_runs(size_t points, size_t clusters) { return points / CE_RUN + clusters; }

// Batch-wide prefix offsets of up to three per-frame counters, made by the last
// CTA of the kernel that writes the counters.
struct BatchOffsets {
    uint32_t which[3];
    uint32_t* offsets[3];  // n_frames + 1 entries each, or null
    uint32_t* ticket;      // CTAs that have finished; zero before the kernel
};

struct PipelineParams {
    int min_white_black_diff;
    uint32_t min_component_size;
    uint32_t min_cluster_pixels;
    uint32_t tag_width;
    int normal_border, reversed_border;
    float max_line_fit_mse;
    float cos_critical_f;      // float(cos(angle)) for do_indexing
    double cos_critical_d;     // cos(angle) for the corner check
    double min_area;           // 0.95 * min_tag_width^2
    int compat_peak_index;
};

// k_pixels.cu
__global__ void k_decimate(const __grid_constant__ FrameSet fs);
__global__ void k_threshold(const __grid_constant__ FrameSet fs, int min_diff, int write_extrema);
__global__ void k_threshold_overlapped(const __grid_constant__ FrameSet fs, int min_diff, int write_extrema);
// CCL tiles of 32 x 8 or 32 x 16 blocks (2x2 pixels)
__global__ void k_ccl_local_r8(const __grid_constant__ FrameSet fs);
__global__ void k_ccl_local_r8_overlapped(const __grid_constant__ FrameSet fs);
__global__ void k_ccl_local_r16(const __grid_constant__ FrameSet fs);
__global__ void k_ccl_local_r16_overlapped(const __grid_constant__ FrameSet fs);
__global__ void k_ccl_local_stage(const __grid_constant__ FrameSet fs);  // r16 over a caller's image: any byte values
__global__ void k_ccl_local_r32(const __grid_constant__ FrameSet fs);
__global__ void k_ccl_local_r32_overlapped(const __grid_constant__ FrameSet fs);
__global__ void k_ccl_border_r16(const __grid_constant__ FrameSet fs);
__global__ void k_ccl_border_edges_r8(const __grid_constant__ FrameSet fs);
__global__ void k_ccl_border_edges_r8_overlapped(const __grid_constant__ FrameSet fs);
__global__ void k_ccl_border_edges_r16(const __grid_constant__ FrameSet fs);
__global__ void k_ccl_border_edges_r16_overlapped(const __grid_constant__ FrameSet fs);
__global__ void k_ccl_border_edges_r32(const __grid_constant__ FrameSet fs);
__global__ void k_ccl_border_edges_r32_overlapped(const __grid_constant__ FrameSet fs);
// final labelling: grid (cdiv(w / 4, CCL_FINAL_THREADS), h / 2, frames) of
// CCL_FINAL_THREADS threads, one pair of 2x2 blocks per thread
constexpr int CCL_FINAL_THREADS = 128;
__global__ void k_ccl_final(const __grid_constant__ FrameSet fs);
__global__ void k_ccl_final_overlapped(const __grid_constant__ FrameSet fs);
__global__ void k_boundaries_dense(const __grid_constant__ FrameSet fs, uint32_t min_size);

// k_quads.cu (drop-in stage kernels)
__global__ void k_fit_lines_windowed(const atag_line_fit_point* points, const uint16_t* cluster_indices,
                                     const atag_cluster_extents* extents, size_t n, atag_corner* found);
__global__ void k_do_indexing(const atag_peak_extents* extents, size_t count, const atag_corner* corners,
                              const atag_line_fit_point* points, const atag_cluster_extents* cluster_extents,
                              float max_mse, float cos_critical, atag_fitted_quad* fitted);
constexpr uint32_t PQ_CTAS = 8;  // blocks of k_process_quads, one cluster
__global__ void k_process_quads(const atag_fitted_quad* fitted, size_t count, PipelineParams p,
                                atag_quad_corners* out, size_t cap, uint32_t* count_out);

// k_cluster.cu (fused path)
__global__ void k_reset_frames(const __grid_constant__ FrameSet fs, uint32_t* cursors, uint32_t n_cursors);
// boundary tiles of 64 x 8 or 64 x 16 pixels
__global__ void k_boundaries_pairs_r8(const __grid_constant__ FrameSet fs, uint32_t min_size);
__global__ void k_boundaries_pairs_r8_overlapped(const __grid_constant__ FrameSet fs, uint32_t min_size);
__global__ void k_boundaries_pairs_r16(const __grid_constant__ FrameSet fs, uint32_t min_size);
__global__ void k_boundaries_pairs_r16_overlapped(const __grid_constant__ FrameSet fs, uint32_t min_size);
__global__ void k_pairs_finalize(const __grid_constant__ FrameSet fs, PipelineParams p, uint32_t small_max, BatchOffsets a);
__global__ void k_scatter_points(const __grid_constant__ FrameSet fs);
__global__ void k_cluster_sort_small(const __grid_constant__ FrameSet fs, const uint32_t* work_offsets,
                                     uint32_t n_frames, uint32_t* work_counter, uint32_t cap);
__global__ void k_cluster_sort_large(const __grid_constant__ FrameSet fs, const uint32_t* work_offsets,
                                     uint32_t n_frames, uint32_t* work_counter, uint32_t cap);
__global__ void k_cluster_lines(const __grid_constant__ FrameSet fs, const uint32_t* run_offsets, uint32_t n_frames);
constexpr uint32_t CE_LINES_SMEM = 4 * 12432;  // four warps' RunSums
__global__ void k_cluster_prefix(const __grid_constant__ FrameSet fs, const uint32_t* run_offsets);
__global__ void k_peaks_scan(const __grid_constant__ FrameSet fs, BatchOffsets a);
__global__ void k_index_quads(const __grid_constant__ FrameSet fs, const uint32_t* work_offsets, uint32_t n_frames,
                              PipelineParams p);
__global__ void k_compact_quads(const __grid_constant__ FrameSet fs);

// k_refine.cu: refinement of the detector's quads in place (optional stage)
__global__ void k_refine_detected(const __grid_constant__ FrameSet fs);

// k_stage_cluster.cu (stage entry points over the dense boundary planes)
__global__ void k_planes_pairs(const __grid_constant__ FrameSet fs, const uint32_t* __restrict__ points,
                               const unsigned long long* __restrict__ keys, uint32_t n);
__global__ void k_planes_scatter(const __grid_constant__ FrameSet fs, const uint32_t* __restrict__ points,
                                 const unsigned long long* __restrict__ keys, uint32_t n);
__global__ void k_stage_cluster_out(const __grid_constant__ FrameSet fs, uint16_t* cluster_indices,
                                    unsigned long long* cluster_keys_out);
// corner peaks (stages 13-15): per-cluster counts, offsets and sorted corners
constexpr uint32_t PK_SORT_CAP = 16384;  // corners of one cluster (at most half its points)
constexpr uint32_t PK_SMEM = PK_SORT_CAP * 8;
__global__ void k_peaks_count(const atag_corner* __restrict__ found, const atag_cluster_extents* __restrict__ ext,
                              uint32_t n_clusters, uint32_t* __restrict__ counts);
__global__ void k_peaks_offsets(const uint32_t* __restrict__ counts, uint32_t n_clusters,
                                uint32_t* __restrict__ offsets, atag_peak_extents* __restrict__ peak_extents,
                                uint32_t extents_cap, uint32_t corner_cap, uint32_t* __restrict__ d_counts);
__global__ void k_peaks_sort(const atag_corner* __restrict__ found, const atag_cluster_extents* __restrict__ ext,
                             uint32_t n_clusters, const uint32_t* __restrict__ counts,
                             const uint32_t* __restrict__ offsets, atag_corner* __restrict__ out,
                             uint32_t corner_cap, uint32_t* __restrict__ d_counts);

}  // namespace atag

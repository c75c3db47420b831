// Internal declarations shared by the host-side translation units of libbpgb300.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <string>
#include <vector>

#include "backprojector_gb300.h"

namespace bpgb {

// ---- errors -----------------------------------------------------------------
int set_error(int status, const std::string &msg);  // records msg, returns status
int cuda_error(cudaError_t e, const char *what);    // maps a CUDA error to a status
void clear_error();
void count_launches(uint64_t n);

#define BPGB_CUDA_TRY(expr)                                   \
    do {                                                      \
        cudaError_t e_ = (expr);                              \
        if (e_ != cudaSuccess) return ::bpgb::cuda_error(e_, #expr); \
    } while (0)

// Checks that a GB300-class device (compute capability 10.x) is current.
int require_device(int *sm_count = nullptr);

// cuTensorMapEncodeTiled from the driver (looked up once, no libcuda link needed), or
// null when the driver does not provide it.
using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                   const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                   const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion,
                                   CUtensorMapFloatOOBfill);
EncodeTiledFn tensor_map_encoder();

// Raises (never lowers) a kernel's dynamic shared memory limit on the current device to
// at least `bytes`.  Plans and batches that share a kernel function stay launchable
// whatever order they were created in.
int reserve_dynamic_smem(const void *kernel, uint32_t bytes);

// ---- volume description -------------------------------------------------------
struct Volume {
    uint32_t n[3];
    float zero[3];
    float inc[9];  // rows: x step, y step, z step
    uint64_t count() const { return (uint64_t)n[0] * n[1] * n[2]; }
};

struct BinParams {
    float t0;
    float dT;
    uint32_t T;
};

// ---- exact kernels (bp_exact.cu) ----------------------------------------------
// Bound (bins) on the distance between the kernel's cheap quotient and the reference's over
// a plan's pairs and voxels; 0.5 where none holds (every update is then evaluated in full).
struct ExactFilter {
    float error = 0.5f;
    bool inside = false;  // every bin of the plan lies in [0, T)
};
ExactFilter exact_filter(const bpgb_pair *pairs, uint64_t P, const Volume &vol,
                         const BinParams &bp);
// A plan's kernel and launch shape.
struct ExactShape {
    bool direct = false;  // the reference's expression for every update, no cheap quotient
    uint32_t tile[3] = {1, 1, 1}, tiles[3] = {0, 0, 0}, threads = 0;
    uint32_t splits = 1;  // CTAs that share a tile's pairs (1..16); above 1 d_partial holds that
                          // many volumes
    uint64_t ctas = 0;    // tiles x splits
};
ExactShape exact_shape(const Volume &vol, uint64_t P, const ExactFilter &filter, int sm_count);
// H rows of `pitch` elements, float or interleaved complex64 (is_complex).
int launch_exact(const void *d_H, bool is_complex, uint64_t pitch, const bpgb_pair *d_pairs,
                 uint64_t P, const Volume &vol, const BinParams &bp, const ExactFilter &filter,
                 const ExactShape &shape, void *d_partial, void *d_out, cudaStream_t stream);
int launch_exact_bins(const bpgb_pair *d_pairs, uint64_t P, const Volume &vol,
                      const BinParams &bp, const int64_t *d_ids, int64_t n, int32_t *d_bins,
                      cudaStream_t stream);

// ---- geometry analysis (plan.cpp) ---------------------------------------------
enum Geometry { GEOM_GENERIC = 0, GEOM_SINGLE_LASER = 1, GEOM_EXHAUSTIVE = 2, GEOM_CONFOCAL = 3 };

struct Factorization {
    Geometry geom = GEOM_GENERIC;
    uint64_t L = 0, S = 0;  // pairs p = l * S + s
};
Factorization factorize_pairs(const bpgb_pair *pairs, uint64_t P);

// Orthonormal frame of the voxel basis: rows u[0..2] and the step lengths h[0..2].
// Returns false when the basis is not orthogonal (then only EXACT applies).
bool volume_frame(const Volume &vol, double u[3][3], double h[3]);

// Every pair value, the volume origin / steps, t0 and deltaT are finite (deltaT != 0);
// otherwise *why names the first offender.
bool finite_geometry(const bpgb_pair *pairs, uint64_t P, const Volume &vol,
                     const BinParams &bp, std::string *why);

// ---- fast kernels (bp_fast.cu) ------------------------------------------------
struct FastConfig {
    // lane layout inside a warp (product 32), voxels per thread (k) on a line along
    // axis `kaxis`, consumer warp layout
    uint32_t lx, ly, lz, k, wx, wy, wz, kaxis;
    uint32_t chunk;   // SPAD rows per pipeline stage and tile (<= 64 / groups)
    uint32_t stages;  // pipeline depth
    uint32_t groups = 1;  // tiles per CTA, each with its own wx x wy x wz consumer warps
    uint32_t tile(int a) const {
        const uint32_t l = a == 0 ? lx : (a == 1 ? ly : lz);
        const uint32_t w = a == 0 ? wx : (a == 1 ? wy : wz);
        return l * w * ((uint32_t)a == kaxis ? k : 1);
    }
    uint32_t consumer_warps() const { return wx * wy * wz; }  // per tile
    uint32_t cta_consumer_warps() const { return wx * wy * wz * groups; }
};

// Tile presets; index -1 selects the tuned default for the geometry.
FastConfig fast_preset(int index, int dtype);
int fast_preset_count();

struct FastPlan;  // opaque, defined in bp_fast.cu
// Tables are built on the GPU in FP64 from the plan's device pair list d_pairs (the
// host list was already factorised into fz).
int fast_plan_build(FastPlan **out, const bpgb_pair *d_pairs, uint64_t P,
                    const Factorization &fz, const Volume &vol, const BinParams &bp,
                    const bpgb_options &opt, int sm_count, std::string *why_not);
int fast_plan_execute(FastPlan *fp, const void *d_H, void *d_out, cudaStream_t stream);
// A plan's pass in `parts` launches over consecutive pair splits (and so, in these plans, over
// consecutive rows of H), which may run as the rows arrive: part k needs the first
// fast_plan_part_rows(k) rows; fast_plan_reduce follows all of them.
constexpr uint32_t kMaxParts = 4;
uint32_t fast_plan_parts(const FastPlan *fp);  // the most that make sense (1: run it whole)
uint64_t fast_plan_part_rows(const FastPlan *fp, uint32_t part, uint32_t parts);
int fast_plan_execute_part(FastPlan *fp, const void *d_H, void *d_out, uint32_t part, uint32_t parts,
                           cudaStream_t stream);
int fast_plan_reduce(FastPlan *fp, void *d_out, cudaStream_t stream);
int fast_plan_dump_bins(FastPlan *fp, const int64_t *d_ids, int64_t n, int32_t *d_bins,
                        cudaStream_t stream);
int fast_plan_execute_tiles(FastPlan *fp, const void *d_H, void *d_out, const uint32_t *d_list,
                            const uint32_t *d_count, uint32_t max_tiles, cudaStream_t stream,
                            const float *d_absmax = nullptr, float target = 0.0f);
int fast_plan_select_tiles(FastPlan *fp, const float *d_score, const uint32_t *block_dims,
                           uint32_t block_size, float threshold, uint32_t *d_list,
                           uint32_t *d_count, cudaStream_t stream);
int fast_plan_select_tiles_topk(FastPlan *fp, const float *d_score, const uint32_t *block_dims,
                                uint32_t block_size, uint32_t k, uint32_t *d_list,
                                uint32_t *d_count, cudaStream_t stream);
void fast_plan_info(const FastPlan *fp, bpgb_plan_info *info);
int fast_plan_tables(const FastPlan *fp, float *host_out, uint64_t capacity, uint64_t *count);
int fast_plan_check(FastPlan *fp, uint64_t *violations, uint64_t *timeouts);
void fast_plan_free(FastPlan *fp);
int wait_timeout_probe(uint32_t limit, int *timed_out);

// bpgb_plan_execute_tiles and bpgb_upsample_trilinear with the stored rows' factor
// (*d_absmax / target, as bpgb_volume_scale) applied to what they write; the tile list needs a
// plan with pair splits, whose reduction applies it.
int plan_execute_tiles_scaled(bpgb_plan plan, const void *d_H, void *d_volume,
                              const uint32_t *d_tile_list, const uint32_t *d_tile_count,
                              uint32_t max_tiles, const float *d_absmax, float target,
                              cudaStream_t stream);
int upsample_scaled(const float *d_coarse, const uint32_t *coarse_dims, float *d_fine,
                    const uint32_t *fine_dims, const float *d_absmax, float target,
                    cudaStream_t stream);

// ---- phasor (phasor.cu) -------------------------------------------------------
int launch_phasor_pulse(const float *d_H, uint64_t rows, uint32_t T, uint32_t in_pitch,
                        const float *h_taps, int K, float *d_out, uint32_t out_pitch,
                        cudaStream_t stream);

// ---- geometry kernels (geometry.cu) -------------------------------------------
int launch_pairs_fp64(const float *d_laser_grid, uint32_t lx, uint32_t ly,
                      const float *d_camera_grid, uint32_t cx, uint32_t cy,
                      const double *laser_pos, const double *camera_pos, int confocal,
                      bpgb_pair *d_out, cudaStream_t stream);

}  // namespace bpgb

// launch.h -- host-side launchers for the step kernels.  Each is explicitly
// instantiated for double in k_f64.cu (built with -fmad=false so FP64 results
// are bit-identical to the CPU restatement) and for float in k_f32.cu.
#pragma once

#include <cuda_runtime.h>

#include "k_common.cuh"
#include "k_dendrite.cuh"
#include "k_dendrite2.cuh"
#include "k_dendrite3.cuh"
#include "k_dendrite_tile.cuh"
#include "k_kh.cuh"
#include "k_kh_strip.cuh"
#include "k_kh_tile.cuh"
#include "k_modelb.cuh"
#include "k_modelb_fast.cuh"
#include "k_modelb_tile.cuh"
#include "k_reduce.cuh"
#include "k_batch.cuh"
#include "k_post.cuh"

namespace dba {

enum { MODEL_DENDRITE = 0, MODEL_MODELB = 1, MODEL_KH = 2 };

template <typename R> bool shape_supported(int model, int D, int B);
template <typename R> int step_grid(int model, int D, int B, int sms);
template <typename R>
cudaError_t launch_dendrite(int D, int B, bool dba_mode, int grid, int sms, cudaStream_t st, const GridP& g, const FlagP& f,
                            const DenP<R>& P);
// FP32 3-D dendrite on double-buffered 32x8x8-cell tiles (k_dendrite_tile.cuh), for grids that
// need a tile list (dendrite3_listed)
// (tile coordinates are packed into 10-bit fields of the tile-queue entry)
inline bool dendrite_tiles_ok(int D, int B, int nx, int ny, int nz)
{
    return D == 3 && B == 8 && (nx + 31) / 32 <= 1024 && ny / 8 <= 1024 && nz / 8 <= 1024;
}
int dendrite3_tile_grid(int sms, int ntiles);
// tiles of the general 3-D dendrite kernel (k_dendrite3.cuh)
inline int dendrite3_tiles(int nx, int ny, int nz) { return ((nx + 31) / 32) * ((ny + 7) / 8) * ((nz + 7) / 8); }
// Whether it works from a list (resident: CTAs on the GPU at once).  The scan is a launch of
// its own; without it each idle tile costs a CTA that reads its flags and ends.
// us per step, list / none: FP64 4^3 blocks 128^3 (2.3 tiles per resident CTA) 18.2 / 15.9,
// 192x160x96 (3.2) 14.4 / 13.8 and 22.3 / 22.0, 256^3 (18) 67.7 / 76.7; FP32 8^3 200x136x104 (2.1)
// 12.6 / 11.7, 18.5 / 18.5; 256x176x128 (3.8) 20.0 / 22.0.
// FP32 8^3 grids that need a list take the double-buffered tiles of k_dendrite_tile.cuh instead (us
// per step against this kernel's list): 512^3 dense 745 / 779; 232^3 21.6 / 23.0 and 48 / 52.
inline bool dendrite3_listed(int tiles, int resident) { return tiles > 4 * resident; }
// 2-D: whether a step goes by tiles (k_dendrite2.cuh): every regular step, and DBA steps up to 5 tiles per
// SM in FP64, 9 in FP32.  us per step, owned / tiles: FP64 864^2 in 32^2 blocks (729 tiles) 8 % active
// 8.1 / 6.3, 17 % 8.3 / 8.7; 512^2 in 8^2 blocks (1024) 5.1 / 5.3; FP32 512^2 in 8^2 blocks
// (1024) 4.9 / 3.7; 1152^2 in 32^2 blocks (1296) 8.3 / 5.0.
inline int dendrite2_tiles(int B, int nx, int ny) { return ((nx + 31) / 32) * (B > 8 ? ny / B : (ny + 7) / 8); }
inline bool dendrite2_tiled(int precision_bytes, bool dba_mode, int tiles, int sms)
{
    return !dba_mode || tiles <= (precision_bytes == 8 ? 5 * sms : 9 * sms);
}
cudaError_t launch_dendrite3_tiles(bool dba_mode, int grid, cudaStream_t st, const GridP& g, const FlagP& f,
                                   const DenP<float>& P);
// FP32 2-D uses the fast kernels (lazy conserved correction, reduction fused):
// the 32x32-cell tile kernel when `tiles` (see modelb_tiles_ok), else one block
// at a time.  `lz` may be null for FP64.
// tiles: 0 modelb_fast_step, 1 the tile kernel with 16-byte cp.async staging, 2 the
// tile kernel with bulk-copy (TMA engine) staging
template <typename R>
cudaError_t launch_modelb(int D, int B, bool dba_mode, int grid, cudaStream_t st, const GridP& g, const FlagP& f,
                          const MBP<R>& P, const LazyP* lz, int tiles);
template <typename R> bool modelb_uses_fast(int D, int B);
bool modelb_tiles_ok(int D, int B, int nx, int ny);
// persistent grid of the tile kernel (also sets its shared-memory limit on the current device)
int modelb_tile_grid(int B, int sms, int ntiles);
cudaError_t launch_modelb_tiles(int B, bool dba_mode, int grid, cudaStream_t st, const GridP& g, const FlagP& f,
                                const MBFastP& P, const MBFastBuf& Q, const LazyP& L, bool bulk);
// ncells: the divisor of the conserved offset (the whole domain's cells; a slab's context
// holds only part of it)
cudaError_t launch_gather_lazy(cudaStream_t st, const GridP& g, int B, const float* b0, const float* b1,
                               const uint8_t* par, const long long* tot_q, const long long* chg_q, size_t count,
                               double ncells, double* out);
template <typename R>
cudaError_t launch_kh(int B, bool dba_mode, int grid, cudaStream_t st, const GridP& g, const FlagP& f, const KHP<R>& P);
template <typename R> cudaError_t launch_correct(int grid, cudaStream_t st, const GridP& g, const CorrP<R>& P);
// one-kernel KH step on 16x16-cell tiles (k_kh_tile.cuh) when kh_tiles_ok
inline bool kh_tiles_ok(int D, int B, int nx, int ny)
{
    return D == 2 && (B == 8 || B == 16) && nx % 16 == 0 && ny % 16 == 0;
}
// Whether its fully active regions go through strips (k_kh_strip.cuh): FP32, and enough cells for
// the strips' warps to fill the GPU.  us per step, DBA with every block active, tiles / strips:
// 512^2 18.6 / 26, 1024^2 36.9 / 30.7, 2048^2 120 / 69.
inline bool kh_strips_ok(int precision_bytes, int nx, int ny) { return precision_bytes == 4 && (long long)nx * ny >= 1 << 20; }
template <typename R> int kh_tile_grid(int B, int sms, int ntiles);
template <typename R>
cudaError_t launch_kh_tile(int B, bool dba_mode, int grid, cudaStream_t st, const GridP& g, const FlagP& f,
                           const KHTileP<R>& P, const KHStripP* X, int sms);   // X: null without strips
// rings of the blocks that the next step finds asleep (k_kh_strip.cuh); f, P: of the next step
cudaError_t launch_kh_strip_flush(int B, cudaStream_t st, const GridP& g, const FlagP& f, const KHTileP<float>& P);
// out[k] = buf[par[owner(cell)]][start + k*stride] for k < count (par may be null -> buffer 0)
template <typename R>
cudaError_t launch_gather(cudaStream_t st, const GridP& g, int B, int D, const R* b0, const R* b1, const uint8_t* par,
                          size_t start, size_t stride, size_t count, double* out);
// KH: recompute primitives from the conserved fields in every block flagged in `only` (all when null)
template <typename R>
cudaError_t launch_kh_prim_blocks(cudaStream_t st, const GridP& g, int B, const KHP<R>& P, const uint8_t* only);

// batched dendrite (k_batch.cuh)
template <typename R> int batch_grid(int B, int threads, int sms);
template <typename R>
cudaError_t launch_batch_step(int B, int threads, int grid, cudaStream_t st, const BatchP& p, const FlagP& f);
// persistent form: `nsteps` steps from step s0 in one cooperative launch (grid from batch_steps_grid)
template <typename R> int batch_steps_grid(int B, int threads, int sms);
template <typename R>
cudaError_t launch_batch_steps(int B, int threads, int grid, cudaStream_t st, const BatchP& p, const BatchFlagBase& fb,
                               long long s0, int nsteps, const GridBar& gb);
template <typename R>
cudaError_t launch_batch_tips(cudaStream_t st, const BatchP& p, const uint8_t* par_cur, int nslots, double* tips);

cudaError_t launch_reduce(cudaStream_t st, const double* bsum, int nb, int nq, double* l1, unsigned int* ticket,
                          double* avg, double ncells);

}  // namespace dba

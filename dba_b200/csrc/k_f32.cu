// FP32 instantiations of the step kernels (stencil arithmetic in float, FMA
// contraction allowed; conserved-change sums stay FP64).
#define REAL_T float
#include <algorithm>

#include "k_inst.cuh"

namespace dba {

cudaError_t launch_gather_lazy(cudaStream_t st, const GridP& g, int B, const float* b0, const float* b1,
                               const uint8_t* par, const long long* tot_q, const long long* chg_q, size_t count,
                               double ncells, double* out)
{
    size_t blocks = (count + kThreads - 1) / kThreads;
    int grid = (int)(blocks < 4096 ? blocks : 4096);
    gather_lazy_kernel<<<grid, kThreads, 0, st>>>(g, B, b0, b1, par, tot_q, chg_q, count, ncells, out);
    return cudaGetLastError();
}

cudaError_t launch_kh_strip_flush(int B, cudaStream_t st, const GridP& g, const FlagP& f, const KHTileP<float>& P)
{
    const int grid = (g.nb + 255) / 256;
    if (B == 8) kh_strip_flush<8><<<grid, 256, 0, st>>>(g, f, P);
    else kh_strip_flush<16><<<grid, 256, 0, st>>>(g, f, P);
    return cudaGetLastError();
}

bool modelb_tiles_ok(int D, int B, int nx, int ny)
{
    // Grids of whole tiles; or of whole blocks, two tiles across and 64 tiles in all: the last tiles
    // then reach past the edge and continue with the first blocks, a single wrap away.  us per
    // step, one block at a time / tiles: 1000 x 760 in 8^2 blocks, 44 % active 20.3 / 10.9, all
    // 30.7 / 10.5; 400 x 272 in 16^2 blocks (117 tiles) 8.9 / 7.3; 200 x 136 in 8^2 blocks (35
    // tiles) 6.2 / 6.6; 1920 x 1600 in 32^2 blocks 59.8 / 28.6.
    if (D != 2 || (B != 8 && B != 16 && B != 32)) return false;
    constexpr int T = MBTile<16>::T;
    return (nx % T == 0 && ny % T == 0) || (nx >= 2 * T && ny >= 2 * T && (long long)nx * ny >= 64 * T * T);
}

template <int B>
static int tile_grid_b(int sms, int ntiles)
{
    const size_t sm = MBTile<B>::smem;
    auto allow = [&](auto kernel) { cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm); };
    allow(modelb_tile_step<B, kMBTileRows, true, false, false>);
    allow(modelb_tile_step<B, kMBTileRows, false, false, false>);
    allow(modelb_tile_step<B, kMBTileRows, true, true, false>);
    allow(modelb_tile_step<B, kMBTileRows, false, true, false>);
    if constexpr (B < 32) {
        allow(modelb_tile_step<B, kMBTileRows, true, false, true>);
        allow(modelb_tile_step<B, kMBTileRows, false, false, true>);
        allow(modelb_tile_step<B, kMBTileRows, true, true, true>);
        allow(modelb_tile_step<B, kMBTileRows, false, true, true>);
    }
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, modelb_tile_step<B, kMBTileRows, true, false, false>, MBTile<B>::NT,
                                                      sm) != cudaSuccess ||
        occ < 1)
        occ = 1;
    const int g = occ * sms;
    return g < ntiles ? g : ntiles;
}

int dendrite3_tile_grid(int sms, int ntiles)
{
    const size_t sm = DenTile::smem;
    cudaFuncSetAttribute(dendrite3_tile_step<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    cudaFuncSetAttribute(dendrite3_tile_step<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, dendrite3_tile_step<true>, DenTile::NT, sm) != cudaSuccess ||
        occ < 1)
        occ = 1;
    const int g = occ * sms;
    return g < ntiles ? g : ntiles;
}

cudaError_t launch_dendrite3_tiles(bool dba_mode, int grid, cudaStream_t st, const GridP& g, const FlagP& f,
                                   const DenP<float>& P)
{
    if (!f.tlist || !f.tctr) return cudaErrorInvalidValue;
    // the scan lists the step's tiles (one thread per block), the tile kernel takes them
    const int sg = (int)std::min<long long>(((long long)g.nb + 255) / 256, 65535);
    const cudaError_t e = launch_beside(dba_mode ? dendrite3_tile_scan<true> : dendrite3_tile_scan<false>, sg, 256, 0, st, g, f);
    if (e != cudaSuccess) return e;
    return launch_beside(dba_mode ? dendrite3_tile_step<true> : dendrite3_tile_step<false>, grid, DenTile::NT, DenTile::smem, st, g, f, P);
}

int modelb_tile_grid(int B, int sms, int ntiles)
{
    return B == 8 ? tile_grid_b<8>(sms, ntiles) : (B == 16 ? tile_grid_b<16>(sms, ntiles) : tile_grid_b<32>(sms, ntiles));
}

template <int B, bool RAG>
static cudaError_t modelb_tiles(bool dba_mode, bool bulk, int grid, cudaStream_t st, const GridP& g, const FlagP& f,
                                const MBFastP& P, const MBFastBuf& Q, const LazyP& L)
{
    const MBPairP K = make_pair_params(P);
    const size_t sm = MBTile<B>::smem;
    const int nt = MBTile<B>::NT;
    auto kernel = bulk ? (dba_mode ? modelb_tile_step<B, kMBTileRows, true, true, RAG> : modelb_tile_step<B, kMBTileRows, false, true, RAG>)
                       : (dba_mode ? modelb_tile_step<B, kMBTileRows, true, false, RAG> : modelb_tile_step<B, kMBTileRows, false, false, RAG>);
    return launch_beside(kernel, grid, nt, sm, st, g, f, P, K, Q, L);
}

cudaError_t launch_modelb_tiles(int B, bool dba_mode, int grid, cudaStream_t st, const GridP& g, const FlagP& f,
                                const MBFastP& P, const MBFastBuf& Q, const LazyP& L, bool bulk)
{
    const bool rag = g.nx % 32 != 0 || g.ny % 32 != 0;
    if (B == 8)
        return rag ? modelb_tiles<8, true>(dba_mode, bulk, grid, st, g, f, P, Q, L)
                   : modelb_tiles<8, false>(dba_mode, bulk, grid, st, g, f, P, Q, L);
    if (B == 16)
        return rag ? modelb_tiles<16, true>(dba_mode, bulk, grid, st, g, f, P, Q, L)
                   : modelb_tiles<16, false>(dba_mode, bulk, grid, st, g, f, P, Q, L);
    if (B == 32) return modelb_tiles<32, false>(dba_mode, bulk, grid, st, g, f, P, Q, L);
    return cudaErrorInvalidValue;
}

}  // namespace dba

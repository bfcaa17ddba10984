// k_reduce.cuh -- conserved-DBA global change and its correction.
//
// The reference's conserved variants (example_Reactive_ModelB/Conserved/kernel.cu:1152-1165,
// example_Kelvin_Helmholtz/Conserved/KH_DBA.cu:1553-1575) store the per-cell
// change of every conserved field (zero in inactive blocks), sum each over
// the whole grid with thrust::reduce (a host round trip per field), divide by
// the cell count and subtract the mean from every cell (Conservation,
// Conserved/kernel.cu:526-553, Conserved/KH_DBA.cu:1366-1392).
//
// Here the step kernel already left one FP64 sum per block (fixed tree over
// the block's cells).  cons_reduce sums those per-block values in a fixed
// order -- a 1024-wide tree (warp shuffles, strides 16..1, then across the 32
// warps) over each run of 1024 blocks, then the same tree over the run sums,
// done by the last CTA to finish (one atomic ticket) -- and writes the means to
// device memory, so no host round trip is needed.  cons_correct then applies
// them to every cell of the block's current buffer.
#pragma once

#include "k_common.cuh"

namespace dba {

// the tree of up to 4 fields side by side, one value of each per thread of a 1024-thread CTA:
// field q's total in lane 0 of warp q
__device__ __forceinline__ double tree1024(double v[4], int nq, double (*s32)[32])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (q >= nq) break;
#pragma unroll
        for (int h = 16; h >= 1; h /= 2) v[q] += __shfl_down_sync(0xffffffffu, v[q], h);
        if (lane == 0) s32[q][warp] = v[q];
    }
    __syncthreads();
    double t = 0.0;
    if (warp < nq) {
        t = s32[warp][lane];
#pragma unroll
        for (int h = 16; h >= 1; h /= 2) t += __shfl_down_sync(0xffffffffu, t, h);
    }
    __syncthreads();
    return t;
}

// grid: J = ceil(nb/1024) CTAs of 1024 threads.  bsum [nq][nb] -> l1 [nq][J];
// the last CTA writes avg[q] = total_q / ncells.  Latency is all there is to it: the fields
// go through the two trees together, one round trip to memory per level.
static __global__ void __launch_bounds__(1024) cons_reduce(const double* bsum, int nb, int nq, double* l1, int J,
                                                    unsigned int* ticket, double* avg, double ncells)
{
    __shared__ double s32[4][32];
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    grid_wait();                                 // the step's kernels
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    const long long i = (long long)blockIdx.x * 1024 + threadIdx.x;
    for (int q = 0; q < nq; ++q) v[q] = i < nb ? bsum[(size_t)q * nb + i] : 0.0;
    double t = tree1024(v, nq, s32);
    if (gridDim.x == 1) {                        // the second tree would add zeros
        if (warp < nq && lane == 0) avg[warp] = (t + 0.0) / ncells;
        return;
    }
    if (warp < nq && lane == 0) {
        l1[(size_t)warp * J + blockIdx.x] = t;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();                         // the other warps' totals, seen at the barrier, before the ticket
        unsigned prev = atomicAdd(ticket, 1u);
        s_last = (prev == gridDim.x - 1);
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // J <= 1024 per level-1 run; zero padding to 1024 leaves the tree's sum unchanged
    for (int q = 0; q < nq; ++q) v[q] = threadIdx.x < J ? ((volatile double*)l1)[(size_t)q * J + threadIdx.x] : 0.0;
    t = tree1024(v, nq, s32);
    if (warp < nq && lane == 0) avg[warp] = t / ncells;
    if (threadIdx.x == 0) *ticket = 0u;
}

// every cell of the block's current buffer: f -= avg (field slot map: bsum
// slot q corrects field map[q])
template <typename R>
struct CorrP {
    R* f[4][2];          // field, buffer (buffer 1 unused when par == nullptr)
    int map[4];
    int nq;
    const uint8_t* par;  // current buffer per block, or nullptr for in-place state
    int B, D;
    const double* avg;
};

// One 16-byte piece of every field per thread (a piece lies in one block: the block edge is a
// multiple of its cells).  The form before took one cell per thread and five 64-bit divisions
// to find its block.
// Reduction and correction, 768^2 FP64 Model B step 52.6 -> 48.9 us, 256 x 200 23.4 -> 19.4,
// 512^2 FP64 KH 56.8 -> 50.9.
template <typename R>
__global__ void __launch_bounds__(kThreads) cons_correct(GridP g, CorrP<R> P)
{
    constexpr int PC = 16 / (int)sizeof(R);
    struct alignas(16) Piece { R v[PC]; };
    const int npr = g.nx / PC;                   // pieces per row
    const unsigned np = (unsigned)npr * g.ny * g.nz;
    grid_wait();                                 // cons_reduce
    double a[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) a[q] = q < P.nq ? P.avg[q] : 0.0;
    for (unsigned i = blockIdx.x * kThreads + threadIdx.x; i < np; i += gridDim.x * kThreads) {
        int buf = 0;
        if (P.par) {
            const int r = (int)(i / (unsigned)npr), x = (int)(i - (unsigned)r * npr) * PC;
            const int z = P.D == 3 ? r / g.ny : 0, y = r - z * g.ny;
            buf = P.par[x / P.B + g.nbx * (y / P.B + g.nby * (P.D == 3 ? z / P.B : 0))];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (q >= P.nq) break;
            const int k = P.map[q];
            Piece* f = reinterpret_cast<Piece*>(buf ? P.f[k][1] : P.f[k][0]) + i;
            Piece p = *f;
#pragma unroll
            for (int e = 0; e < PC; ++e) p.v[e] = (R)((double)p.v[e] - a[q]);
            *f = p;
        }
    }
}

}  // namespace dba

// k_dendrite3.cuh -- 3-D dendrite step over tiles of 32 x 8 x 8 cells: FP64, FP32 in 4^3 blocks,
// and small FP32 grids in 8^3 blocks (large ones: k_dendrite_tile.cuh).
//
// Same DBA semantics as every dendrite kernel; point arithmetic in k_dendrite.cuh.  A scan kernel
// does the step's block bookkeeping and lists the tiles that have an active block, with
// their blocks' activity and parity; the CTAs of the tile kernel, a few times as many as
// are resident, step through the list (small grids: no list, a CTA per tile).  Per tile:
//   * p and T of the tile plus one cell are staged as 16-byte pieces, each inside one block
//     whose parity picks the buffer, and only in blocks that are active or share a face with
//     an active block of the tile; a thread keeps one piece of a plane and steps over planes;
//   * the warps take the active blocks in turn, those active in p first: a p update is a
//     chain of about 50 FP64 operations and two divisions, a T update one of 10, and with
//     a fixed share of the tile per warp the others waited for the warp that held the front;
//   * a cell at a zero-flux wall is its own neighbour, so nothing is staged beyond a wall; a
//     tile away from the walls has its neighbours at constant offsets of the loads.
// What bounds it: the table and staging round trips of a thin active shell, which the
// resident CTAs hide for each other (three per SM in FP64, five in FP32), and
// instruction issue.  The kernel before worked on one 4^3 block of 64 cells per quarter CTA
// and staged 216 cells for it, each with its own index arithmetic.  Measured on the way
// and dropped: CTAs that stay and take tiles from a counter two ahead, 70.7 against 67.7 us
// (fewer round trips per tile, but fewer CTAs in flight).
// Measured per step, before -> now: 256^3 FP64 in 4^3 blocks (16 % p-, 44 % T-active) 214 ->
// 66.4 us, in 8^3 blocks 116 -> 70; 200 x 136 x 104 FP32 in 8^3 blocks, every block,
// 42.7 -> 24.6, in 4^3 blocks 84.9 -> 28.5.  A grid that is nearly all asleep was faster one block
// at a time: 128^3 FP64 0.6 % p-active 7.7 -> 9.9, 4 % 16.5 -> 12.1.
#pragma once

#include "k_common.cuh"
#include "k_dendrite.cuh"

namespace dba {

constexpr int kDenEntry = 8;                             // ints per entry of the tile list

template <typename R, int B>
struct Den3 {
    static constexpr int NT = 256;
    static constexpr int TX = 32, TY = 8, TZ = 8;
    static constexpr int V = B * B * B;
    static constexpr int NBX = TX / B, NBY = TY / B, NBZ = TZ / B, NBT = NBX * NBY * NBZ;
    static constexpr int RX = NBX + 2, RY = NBY + 2, RZ = NBZ + 2, NR = RX * RY * RZ;
    static constexpr int PC = 16 / (int)sizeof(R);       // cells per staged piece
    // row and plane pitch (column x at x + PC): the row segments of a warp's cells fall on distinct banks
    static constexpr int SP = sizeof(R) == 8 && B == 4 ? 36 : 40;
    static constexpr int SH = TY + 2, SD = TZ + 2, PL = SP * SH + (sizeof(R) == 4 && B == 4 ? 4 : 0), SV = PL * SD;
    // Work items of a warp, one block or part of it (IPB items per block), NZ cells per lane:
    // a block of 4^3 as 4 x 4 columns and planes z, z + 2; of a block of 8^3 8 x 4 columns
    // and 8 planes (FP32) or 4 (FP64, where a cell is a long chain)
    static constexpr int NZ = B == 4 ? 2 : (sizeof(R) == 8 ? 4 : 8), DZ = B == 4 ? 2 : 1;
    static constexpr int IPB = V / (32 * NZ);
    static constexpr int NPR = TX / PC + 2;              // pieces per staged row: x from -PC to TX + PC - 1
    static constexpr int PP = NPR * SH, ZP = NT / PP;    // pieces of a plane, planes staged at once
    static constexpr size_t smem = sizeof(R) * 2 * SV;
    static constexpr int MINB = sizeof(R) == 8 ? 3 : 5;  // resident CTAs per SM
    static_assert(ZP >= 1 && NBT <= 32 && (NBT & (NBT - 1)) == 0 && TX % B == 0 && 8 % B == 0 && B % PC == 0 && 4 % PC == 0, "tile shape");
};

// Block bookkeeping of one step, a thread per block, a tile's blocks on adjacent lanes of one
// warp (all its lanes call): parity flip of active blocks, clearing of the flag array two
// steps ahead, activity counts.  Returns the tile's masks: blocks active in p, in T,
// parity in p, in T.  (x, y, z) the tile, k the thread's block in it; in: the tile exists.
template <typename S, bool DBA>
__device__ __forceinline__ uint4 den_blocks(const GridP& g, const FlagP& f, bool in, int tx, int ty, int tz, int k)
{
    constexpr int NBT = S::NBT;
    const int nb = g.nb;
    const int x = tx * S::NBX + k % S::NBX, y = ty * S::NBY + (k / S::NBX) % S::NBY, z = tz * S::NBZ + k / (S::NBX * S::NBY);
    const bool valid = in && x < g.nbx && y < g.nby && z < g.nbz;
    int act = 0, pp = 0, pT = 0;
    if (valid) {
        const int b = x + g.nbx * (y + g.nby * z);
        pp = f.par_cur[b];
        pT = f.par_cur[nb + b];
        act = DBA ? ((f.wake_cur[b] ? 1 : 0) | (f.wake_cur[nb + b] ? 2 : 0)) : 3;
        f.wake_clr[b] = 0;
        f.wake_clr[nb + b] = 0;
        if (!DBA) {
            f.wake_nxt[b] = 1;
            f.wake_nxt[nb + b] = 1;
        }
        f.par_nxt[b] = (uint8_t)(pp ^ (act & 1));
        f.par_nxt[nb + b] = (uint8_t)(pT ^ (act >> 1));
    }
    count_stats(f.stats, act, valid);
    const int g0 = (threadIdx.x & 31) & ~(NBT - 1);
    const unsigned gm = NBT == 32 ? 0xffffffffu : (1u << NBT) - 1u;
    uint4 m;
    m.x = (__ballot_sync(0xffffffffu, act & 1) >> g0) & gm;
    m.y = (__ballot_sync(0xffffffffu, act & 2) >> g0) & gm;
    m.z = (__ballot_sync(0xffffffffu, pp != 0) >> g0) & gm;
    m.w = (__ballot_sync(0xffffffffu, pT != 0) >> g0) & gm;
    return m;
}

// Scan of one step: the bookkeeping, and one list entry per tile with an active block: [0]
// its x, [1..4] its masks, [5] [6] its y and z (in tiles).
template <typename S, bool DBA>
__global__ void __launch_bounds__(256) dendrite_scan(GridP g, FlagP f, int ntiles)
{
    const int lane = threadIdx.x & 31;
    const int ntx = (g.nx + S::TX - 1) / S::TX, nty = (g.ny + S::TY - 1) / S::TY;
    const int it = blockIdx.x * 256 + threadIdx.x;       // the grid covers ntiles * NBT items
    const int tile = it / S::NBT, k = it % S::NBT;
    const int tx = tile % ntx, ty = (tile / ntx) % nty, tz = tile / (ntx * nty);
    grid_wait();                                         // the step before
    const uint4 m = den_blocks<S, DBA>(g, f, tile < ntiles, tx, ty, tz, k);
    const bool take = k == 0 && (m.x | m.y) != 0;
    const unsigned mt = __ballot_sync(0xffffffffu, take);
    if (mt == 0) return;
    unsigned base = 0;
    if (lane == __ffs(mt) - 1) base = atomicAdd(f.tctr, (unsigned)__popc(mt));
    base = __shfl_sync(0xffffffffu, base, __ffs(mt) - 1);
    if (take) {
        const unsigned e = base + (unsigned)__popc(mt & ((1u << lane) - 1u));
        if (e < (unsigned)ntiles) {
            int* d = f.tlist + (size_t)e * kDenEntry;
            *reinterpret_cast<int4*>(d) = make_int4(tx, (int)m.x, (int)m.y, (int)m.z);
            *reinterpret_cast<int4*>(d + 4) = make_int4((int)m.w, ty, tz, 0);
        }
    }
}

// One work item: block k of the tile (activity pa, Ta), part sub.  EDGE: the tile touches a
// zero-flux wall, where a cell is its own neighbour (offset 0); elsewhere the offsets are
// constants of the loads.  sp, sT: the staged tile; po, to: the destination buffers at
// the tile's first cell.  Returns bit 0 / 1: a cell passes the p / T wake-up test, bit 2: a
// stored value is not finite.
template <typename R, int B, bool DBA, bool EDGE>
__device__ __forceinline__ unsigned den3_item(const GridP& g, const DenP<R>& P, const R* sp, const R* sT, int k, int sub,
                                              bool pa, bool Ta, int X0, int Y0, int Z0, R* po, R* to)
{
    using S = Den3<R, B>;
    constexpr int SP = S::SP, PL = S::PL, NZ = S::NZ, DZ = S::DZ;
    const int lane = threadIdx.x & 31;
    const int cx = (k % S::NBX) * B + lane % B;
    const int cy = ((k / S::NBX) % S::NBY) * B + (B == 4 ? (lane >> 2) & 3 : 4 * (sub & 1) + (lane >> 3));
    const int cz = (k / (S::NBX * S::NBY)) * B + (B == 4 ? lane >> 4 : NZ * (sub >> 1));
    int dxm = -1, dxp = 1, dym = -SP, dyp = SP;
    if (EDGE) {
        if (X0 + cx == 0) dxm = 0;
        if (X0 + cx == g.nx - 1) dxp = 0;
        if (Y0 + cy == 0) dym = 0;
        if (Y0 + cy == g.ny - 1) dyp = 0;
    }
    const size_t nxy = (size_t)g.nx * g.ny;
    const size_t g0 = (size_t)cx + (size_t)g.nx * cy + nxy * cz;
    po += g0;
    to += g0;
    const R* qp = sp + (cz + 1) * PL + (cy + 1) * SP + cx + S::PC;
    const R* qT = sT + (cz + 1) * PL + (cy + 1) * SP + cx + S::PC;
    auto below = [&](int c) { return EDGE && Z0 + cz + c * DZ == 0 ? 0 : -PL; };
    auto above = [&](int c) { return EDGE && Z0 + cz + c * DZ == g.nz - 1 ? 0 : PL; };
    R pm = qp[below(0)], pc = qp[0], Tm = qT[below(0)], Tc = qT[0];
    bool hp = false, hT = false, bad = false;
    constexpr int U = DZ == 1 && sizeof(R) == 4 ? 2 : NZ;
#pragma unroll U
    for (int c = 0; c < NZ; ++c) {
        const R pq = qp[above(c)], Tq = qT[above(c)];
        R pn = pc;
        if (pa) {                                        // Evolve_p (kernel.cu:220-241)
            if constexpr (sizeof(R) == 4)
                pn = den_p_f32<3>(pc, Tc, qp[dxp], qp[dxm], qp[dyp], qp[dym], pq, pm, P.c32);
            else
                pn = den_p_new<R>(pc, Tc, qp[dxp], qp[dxm], qp[dyp], qp[dym], pq, pm, (R)P.f0, (R)P.f1, (R)P.f2, (R)P.f3,
                                  (R)P.dt, (R)P.delta, (R)P.eps2, (R)P.gamma);
            *po = pn;
            hp |= pn >= (R)P.thr_p && pn <= (R)P.thr_p_hi;
            bad |= !isfinite(pn);
        }
        if (Ta) {                                        // Evolve_T (kernel.cu:286-289, :468-489)
            R Tn;
            if constexpr (sizeof(R) == 4)
                Tn = den_T_f32<3, DBA>(Tc, qT[dxp], qT[dxm], qT[dyp], qT[dym], Tq, Tm, pa, pn, pc, P.c32);
            else
                Tn = den_T_new<R, DBA>(Tc, qT[dxp], qT[dxm], qT[dyp], qT[dym], Tq, Tm, pa, pn, pc, (R)P.f1, (R)P.dt);
            *to = Tn;
            hT |= fabs(Tn - Tc) >= (R)P.thr_T;
            bad |= !isfinite(Tn);
        }
        if (c + 1 == NZ) break;
        qp += DZ * PL;
        qT += DZ * PL;
        po += DZ * nxy;
        to += DZ * nxy;
        if (DZ == 1) {
            pm = pc; pc = pq; Tm = Tc; Tc = Tq;
        } else {
            pm = qp[below(c + 1)]; pc = qp[0]; Tm = qT[below(c + 1)]; Tc = qT[0];
        }
    }
    return (hp ? 1u : 0u) | (hT ? 2u : 0u) | (bad ? 4u : 0u);
}

// LIST: the CTAs step through the scan's list; otherwise CTA b works on tile b of the grid and
// does its bookkeeping itself
template <typename R, int B, bool DBA, bool LIST>
__global__ void __launch_bounds__(256, Den3<R, B>::MINB) dendrite3_step(GridP g, FlagP f, DenP<R> P, int ntiles)
{
    using S = Den3<R, B>;
    constexpr int NT = S::NT, SP = S::SP, PL = S::PL, SV = S::SV;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R* sp = reinterpret_cast<R*>(smem_raw);              // [SD][SH][SP]
    R* sT = sp + SV;
    __shared__ uint8_t s_tab[S::NR];                     // blocks around the tile: bit 0 p parity, 1 T parity, 2 staged
    __shared__ int s_hit[2][2][S::NBT];                  // wake tests by tile parity and channel
    __shared__ uint8_t s_order[S::NBT];                  // the tile's active blocks, those active in p first
    const int tid = threadIdx.x, nb = g.nb, w = tid >> 5;
    __shared__ uint4 s_mask;
    grid_wait();                                         // the scan, or the step before
    const int cnt = LIST ? (int)min(__ldcg(f.tctr), (unsigned)ntiles) : ntiles;
    if (LIST && blockIdx.x == 0 && tid == 0)             // the next step's count: the other of the pair
        *reinterpret_cast<unsigned*>(reinterpret_cast<uintptr_t>(f.tctr) ^ sizeof(unsigned)) = 0u;

    for (int i = blockIdx.x, it = 0; i < cnt; i += gridDim.x, it ^= 1) {
        int4 ea, eb;
        if (LIST) {
            ea = __ldcg(reinterpret_cast<const int4*>(f.tlist + (size_t)i * kDenEntry));
            eb = __ldcg(reinterpret_cast<const int4*>(f.tlist + (size_t)i * kDenEntry + 4));
        } else {
            const int ntx = (g.nx + S::TX - 1) / S::TX, nty = (g.ny + S::TY - 1) / S::TY;
            ea.x = i % ntx; eb.y = (i / ntx) % nty; eb.z = i / (ntx * nty);
            if (tid < 32) {
                const uint4 m = den_blocks<S, DBA>(g, f, tid < S::NBT, ea.x, eb.y, eb.z, tid);
                if (tid == 0) s_mask = m;
            }
            __syncthreads();
            const uint4 m = s_mask;
            if ((m.x | m.y) == 0) continue;              // (the grid has one CTA per tile: i ends here)
            ea.y = (int)m.x; ea.z = (int)m.y; ea.w = (int)m.z; eb.x = (int)m.w;
        }
        const unsigned ap = (unsigned)ea.y, aT = (unsigned)ea.z, pp = (unsigned)ea.w, pT = (unsigned)eb.x, any = ap | aT;
        const int bx0 = ea.x * S::NBX, by0 = eb.y * S::NBY, bz0 = eb.z * S::NBZ;
        const int X0 = ea.x * S::TX, Y0 = eb.y * S::TY, Z0 = eb.z * S::TZ;
        // table of the blocks around the tile, order of its active ones
        if (tid < S::NBT) {
            const unsigned lt = (1u << tid) - 1u;
            if ((any >> tid) & 1u) s_order[(ap >> tid) & 1u ? __popc(ap & lt) : __popc(ap) + __popc(any & ~ap & lt)] = (uint8_t)tid;
            s_hit[it][0][tid] = 0;
            s_hit[it][1][tid] = 0;
        }
        for (int r = tid; r < S::NR; r += NT) {
            const int rx = r % S::RX, ry = (r / S::RX) % S::RY - 1, rz = r / (S::RX * S::RY) - 1;
            auto row = [&](int y, int z) -> unsigned {   // active blocks of a row of the tile, block x at bit x + 1
                return y >= 0 && y < S::NBY && z >= 0 && z < S::NBZ
                           ? ((any >> (S::NBX * (y + S::NBY * z))) & ((1u << S::NBX) - 1u)) << 1 : 0u;
            };
            unsigned m = row(ry, rz);
            m |= (m << 1) | (m >> 1);
            m |= row(ry - 1, rz) | row(ry + 1, rz) | row(ry, rz - 1) | row(ry, rz + 1);
            unsigned v = 0;
            if ((m >> rx) & 1u) {
                int x = bx0 + rx - 1, y = by0 + ry, z = bz0 + rz;
                if (!g.bc) {
                    x = wrap_p(x, g.nbx);
                    y = wrap_p(y, g.nby);
                    z = wrap_p(z, g.nbz);
                }
                // a block beyond a zero-flux wall is not staged
                if (x >= 0 && x < g.nbx && y >= 0 && y < g.nby && z >= 0 && z < g.nbz) {
                    const int b = x + g.nbx * (y + g.nby * z);
                    v = 4u | (f.par_cur[b] ? 1u : 0u) | (f.par_cur[nb + b] ? 2u : 0u);
                }
            }
            s_tab[r] = (uint8_t)v;
        }
        __syncthreads();
        {
            const int ph = tid / S::PP, q = tid - ph * S::PP;
            const int c = q % S::NPR, ry = q / S::NPR;
            const int lx = (c - 1) * S::PC, ly = ry - 1;
            // (a staged block is inside the grid, beyond its edge only where the grid is periodic)
            if (ph < S::ZP && X0 + lx <= g.nx && Y0 + ly <= g.ny) {
                const uint8_t* tr = s_tab + (lx + B) / B + S::RX * ((ly + B) / B);
                const size_t row = (size_t)wrap_p(X0 + lx, g.nx) + (size_t)g.nx * wrap_p(Y0 + ly, g.ny);
                const size_t nxy = (size_t)g.nx * g.ny;
                R* d = sp + ry * SP + lx + S::PC;
#pragma unroll 2
                for (int rz = ph; rz < S::SD; rz += S::ZP) {
                    const unsigned v = tr[S::RX * S::RY * ((rz - 1 + B) / B)];
                    if (!(v & 4u)) continue;
                    if (Z0 + rz - 1 > g.nz) break;
                    const size_t gi = row + nxy * wrap_p(Z0 + rz - 1, g.nz);
                    cp_async16(d + rz * PL, ((v & 1u) ? P.p[1] : P.p[0]) + gi);
                    cp_async16(d + rz * PL + SV, ((v & 2u) ? P.T[1] : P.T[0]) + gi);
                }
            }
            cp_async_commit();
            cp_async_wait0();
        }
        __syncthreads();
        const bool edge = g.bc && (X0 == 0 || Y0 == 0 || Z0 == 0 || X0 + S::TX >= g.nx || Y0 + S::TY >= g.ny || Z0 + S::TZ >= g.nz);
        const int nitem = __popc(any) * S::IPB;
        const size_t base = (size_t)X0 + (size_t)g.nx * ((size_t)Y0 + (size_t)g.ny * Z0);
        for (int j = w; j < nitem; j += NT / 32) {
            const int k = s_order[j / S::IPB], sub = j % S::IPB;
            const bool pa = (ap >> k) & 1u, Ta = (aT >> k) & 1u;
            R* po = ((pp >> k) & 1u ? P.p[0] : P.p[1]) + base;
            R* to = ((pT >> k) & 1u ? P.T[0] : P.T[1]) + base;
            const unsigned r = edge ? den3_item<R, B, DBA, true>(g, P, sp, sT, k, sub, pa, Ta, X0, Y0, Z0, po, to)
                                    : den3_item<R, B, DBA, false>(g, P, sp, sT, k, sub, pa, Ta, X0, Y0, Z0, po, to);
            if (DBA && (r & 1u)) s_hit[it][0][k] = 1;
            if (DBA && (r & 2u)) s_hit[it][1][k] = 1;
            if (r & 4u) raise_status(f.status, 5);
        }
        __syncthreads();
        // wake-up tests and scatter: self + 6 faces per channel (kernel.cu:577-634), neighbour n
        // on warp n, block k on lane k
        const int k = tid & 31;
        if (DBA && w < 7 && k < S::NBT) {
            const int x = bx0 + k % S::NBX, y = by0 + (k / S::NBX) % S::NBY, z = bz0 + k / (S::NBX * S::NBY);
#pragma unroll
            for (int ch = 0; ch < 2; ++ch) {
                if (!(((ch ? aT : ap) >> k) & 1u)) continue;
                const int hit = s_hit[it][ch][k];
                if (w == 0) f.next[(size_t)ch * nb + x + g.nbx * (y + g.nby * z)] = (uint8_t)hit;
                if (hit) {
                    const int nbk = block_nb_k(g, x, y, z, w);
                    if (nbk >= 0) f.wake_nxt[(size_t)ch * nb + nbk] = 1;
                }
            }
        }
    }
}

}  // namespace dba

// k_dendrite2.cuh -- 2-D dendrite step: one CTA per tile of 32 x 8..32 cells (dendrite2_step), or CTAs that
// own scattered blocks (dendrite2_owned, DBA on grids of many tiles).
//
// Same DBA semantics and point arithmetic as the other dendrite kernels (k_dendrite.cuh).  A tile that
// has an active block is staged with one cell around it as 16-byte pieces, each inside one
// block whose parity picks the buffer; a thread owns one to four cells, a warp 8 x 4 of one
// block of 8 and more, so the warps of inactive blocks skip the update; a cell at a
// zero-flux wall is its own neighbour.
//
// What bounds both: latency.  A 512^2 step moves less than 1 MB through L2; its time is the launch
// and the chain flags -> staging -> one cell's formula -> flags.  A tile's CTA reads its flags and
// the parities around it in one round trip and needs three barriers; the owned form needs
// seven per round, but packs active blocks into rounds and has no idle CTAs, which counts
// where most tiles sleep and there are more of them than the GPU holds (dendrite2_tiled).
// us per step, owned / tiles: every block 512^2 FP64 8.2 / 5.9; DBA 512^2 FP32 4.9 / 3.7 (6 % active) and
// 6.2 / 4.4 (16 %), 416^2 FP64 5.8 / 4.2; 512^2 FP64 5.1 / 5.3, 1024^2 FP64 7.6 / 8.5, 1536^2 9.3 / 13
// (with a tile list).  Both since a step's CTAs start as the last ones of the step before end:
// 0.3 to 0.4 us less.
#pragma once

#include <type_traits>

#include "k_common.cuh"
#include "k_dendrite.cuh"
#include "k_dendrite3.cuh"

namespace dba {

template <typename R, int B>
struct Den2 {
    static constexpr int NT = 256;
    static constexpr int TX = 32, TY = B > 8 ? B : 8, TZ = 1;
    static constexpr int NBX = TX / B, NBY = TY / B, NBZ = 1, NBT = NBX * NBY;
    static constexpr int RX = NBX + 2, RY = NBY + 2, NR = RX * RY;
    static constexpr int PC = 16 / (int)sizeof(R);       // cells per staged piece
    static constexpr int SP = 40;                        // row pitch: column x at x + PC
    static constexpr int SH = TY + 2, SV = SP * SH;
    static constexpr int NPR = TX / PC + 2, PP = NPR * SH;   // pieces per staged row, pieces
    static constexpr int NC = TY / 8;                    // cells per thread, 8 rows apart
    static constexpr int MINB = sizeof(R) == 8 ? 5 : 6;  // resident CTAs per SM
    static_assert(NBT <= 32 && (NBT & (NBT - 1)) == 0 && B % PC == 0 && 32 + NR <= NT, "tile shape");
};

// one CTA per tile
template <typename R, int B, bool DBA>
__global__ void __launch_bounds__(256, Den2<R, B>::MINB) dendrite2_step(GridP g, FlagP f, DenP<R> P)
{
    using S = Den2<R, B>;
    constexpr int NT = S::NT, SP = S::SP;
    __shared__ __align__(16) R sp[S::SV], sT[S::SV];
    __shared__ uint8_t s_tab[S::NR];                     // blocks around the tile: bit 0 p parity, 1 T parity
    __shared__ int s_hit[2][S::NBT];                     // wake tests
    __shared__ uint4 s_mask;
    const int tid = threadIdx.x, nb = g.nb, w = tid >> 5, lane = tid & 31;
    const int ntx = (g.nx + S::TX - 1) / S::TX, ty = blockIdx.x / ntx, tx = blockIdx.x - ty * ntx;
    const int X0 = tx * S::TX, Y0 = ty * S::TY;
    grid_wait();                                         // the step before
    if (tid < S::NBT) {
        s_hit[0][tid] = 0;
        s_hit[1][tid] = 0;
    }
    if (tid < 32) {
        const uint4 m = den_blocks<S, DBA>(g, f, tid < S::NBT, tx, ty, 0, tid);
        if (tid == 0) s_mask = m;
    }
    if (tid >= 32 && tid < 32 + S::NR) {             // parities around the tile, beside the flags
        const int r = tid - 32;
        int x = X0 / B + r % S::RX - 1, y = Y0 / B + r / S::RX - 1;
        if (!g.bc) {
            x = wrap_p(x, g.nbx);
            y = wrap_p(y, g.nby);
        }
        // (beyond a zero-flux wall, or past the grid's last tile, nothing is staged)
        if (x >= 0 && x < g.nbx && y >= 0 && y < g.nby) {
            const int b = x + g.nbx * y;
            s_tab[r] = (uint8_t)((f.par_cur[b] ? 1 : 0) | (f.par_cur[nb + b] ? 2 : 0));
        }
    }
    __syncthreads();
    const uint4 m = s_mask;
    const unsigned ap = m.x, aT = m.y, any = ap | aT;
    if (any == 0) return;
    const int vx = min(S::TX, g.nx - X0), vy = min(S::TY, g.ny - Y0);
    for (int q = tid; q < S::PP; q += NT) {
        const int c = q % S::NPR, ry = q / S::NPR, lx = (c - 1) * S::PC, ly = ry - 1;
        int gx = X0 + lx, gy = Y0 + ly;
        if (lx > vx || ly > vy || (g.bc && (gx < 0 || gx >= g.nx || gy < 0 || gy >= g.ny))) continue;
        gx = wrap_p(gx, g.nx);
        gy = wrap_p(gy, g.ny);
        const unsigned v = s_tab[(lx + B) / B + S::RX * ((ly + B) / B)];
        const size_t gi = (size_t)gx + (size_t)g.nx * gy;
        const int so = ry * SP + lx + S::PC;
        cp_async16(sp + so, ((v & 1u) ? P.p[1] : P.p[0]) + gi);
        cp_async16(sT + so, ((v & 2u) ? P.T[1] : P.T[0]) + gi);
    }
    cp_async_commit();
    cp_async_wait0();
    __syncthreads();
    const int cx = 8 * (w & 3) + (lane & 7), cy0 = 4 * (w >> 2) + (lane >> 3);
#pragma unroll
    for (int c = 0; c < S::NC; ++c) {
        const int cy = cy0 + 8 * c, k = cx / B + S::NBX * (cy / B);
        const bool pa = (ap >> k) & 1u, Ta = (aT >> k) & 1u;
        if (!(pa || Ta)) continue;
        const int x = X0 + cx, y = Y0 + cy;
        const int dxm = g.bc && x == 0 ? 0 : -1, dxp = g.bc && x == g.nx - 1 ? 0 : 1;
        const int dym = g.bc && y == 0 ? 0 : -SP, dyp = g.bc && y == g.ny - 1 ? 0 : SP;
        const R* qp = sp + (cy + 1) * SP + cx + S::PC;
        const R* qT = sT + (cy + 1) * SP + cx + S::PC;
        const R pc = qp[0], Tc = qT[0];
        const size_t gi = (size_t)x + (size_t)g.nx * y;
        R pn = pc;
        bool bad = false;
        if (pa) {                                    // Evolve_p (kernel.cu:220-241); the z neighbours are the cell
            if constexpr (sizeof(R) == 4)
                pn = den_p_f32<2>(pc, Tc, qp[dxp], qp[dxm], qp[dyp], qp[dym], pc, pc, P.c32);
            else
                pn = den_p_new<R>(pc, Tc, qp[dxp], qp[dxm], qp[dyp], qp[dym], pc, pc, (R)P.f0, (R)P.f1, (R)P.f2, (R)P.f3,
                                  (R)P.dt, (R)P.delta, (R)P.eps2, (R)P.gamma);
            ((m.z >> k) & 1u ? P.p[0] : P.p[1])[gi] = pn;
            if (DBA && pn >= (R)P.thr_p && pn <= (R)P.thr_p_hi) s_hit[0][k] = 1;
            bad = !isfinite(pn);
        }
        if (Ta) {                                    // Evolve_T (kernel.cu:286-289, :468-489)
            R Tn;
            if constexpr (sizeof(R) == 4)
                Tn = den_T_f32<2, DBA>(Tc, qT[dxp], qT[dxm], qT[dyp], qT[dym], Tc, Tc, pa, pn, pc, P.c32);
            else
                Tn = den_T_new<R, DBA>(Tc, qT[dxp], qT[dxm], qT[dyp], qT[dym], Tc, Tc, pa, pn, pc, (R)P.f1, (R)P.dt);
            ((m.w >> k) & 1u ? P.T[0] : P.T[1])[gi] = Tn;
            if (DBA && fabs(Tn - Tc) >= (R)P.thr_T) s_hit[1][k] = 1;
            bad |= !isfinite(Tn);
        }
        if (bad) raise_status(f.status, 5);
    }
    if (!DBA) return;
    __syncthreads();
    // wake-up tests and scatter: self + 6 faces per channel (kernel.cu:577-634), neighbour n
    // on warp n, block k on lane k (the z faces are the block itself, or a wall)
    if (w < 5 && lane < S::NBT) {
        const int x = X0 / B + lane % S::NBX, y = Y0 / B + lane / S::NBX;
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
            if (!(((ch ? aT : ap) >> lane) & 1u)) continue;
            const int hit = s_hit[ch][lane];
            if (w == 0) f.next[(size_t)ch * nb + x + g.nbx * y] = (uint8_t)hit;
            if (hit) {
                const int nbk = block_nb_k(g, x, y, 0, w);
                if (nbk >= 0) f.wake_nxt[(size_t)ch * nb + nbk] = 1;
            }
        }
    }
}

// CTA c owns blocks c, c + G, ...: it scans their flags 256 at a time, lists the active ones and
// advances them in rounds of 256 cells
template <typename R, int B>
__global__ void __launch_bounds__(kThreads) dendrite2_owned(GridP g, FlagP f, DenP<R> P)
{
    constexpr int NT = kThreads;
    constexpr int V = B * B;
    constexpr int E = B + 2;
    constexpr int TV = E * E;
    constexpr int K = V >= NT ? 1 : NT / V;
    constexpr int CPT = V >= NT ? V / NT : 1;
    constexpr int SY = E;

    __shared__ R sp[K * TV];
    __shared__ R sT[K * TV];
    __shared__ int s_list[NT], s_lmeta[NT];
    __shared__ int s_cnt;
    __shared__ int s_blk[K], s_meta[K], s_np[K], s_nT[K];
    __shared__ int s_bx[K], s_by[K];   // block coordinates of the round's blocks
    static_assert(K * 14 <= NT, "one wake-up scatter thread per block, channel and neighbour");

    const int tid = threadIdx.x;
    const int G = gridDim.x;
    const int nb = g.nb;
    const R f0 = (R)P.f0, f1 = (R)P.f1, f2 = (R)P.f2, f3 = (R)P.f3;
    const R dt = (R)P.dt, delta = (R)P.delta, eps2 = (R)P.eps2, gam = (R)P.gamma;
    const R thr_p = (R)P.thr_p, thr_p_hi = (R)P.thr_p_hi, thr_T = (R)P.thr_T;

    grid_wait();                                         // the step before
    for (long long j0 = 0; blockIdx.x + (long long)G * j0 < nb; j0 += NT) {
        const long long bl = blockIdx.x + (long long)G * (j0 + tid);
        const bool valid = bl < nb;
        const int b = (int)bl;
        int act = 0, meta = 0;
        if (valid) {
            int pp = f.par_cur[b], pT = f.par_cur[nb + b];
            act = (f.wake_cur[b] ? 1 : 0) | (f.wake_cur[nb + b] ? 2 : 0);
            f.wake_clr[b] = 0;
            f.wake_clr[nb + b] = 0;
            f.par_nxt[b] = (uint8_t)(pp ^ (act & 1));
            f.par_nxt[nb + b] = (uint8_t)(pT ^ ((act >> 1) & 1));
            meta = act | (pp << 2) | (pT << 3);
        }
        count_stats(f.stats, act, valid);
        if (tid == 0) s_cnt = 0;
        __syncthreads();
        list_append(valid && act, b, meta, s_list, s_lmeta, &s_cnt);
        __syncthreads();
        const int cnt = s_cnt;

        for (int q0 = 0; q0 < cnt; q0 += K) {
            if (tid < K) {
                int q = q0 + tid;
                const int blk = q < cnt ? s_list[q] : -1;
                s_blk[tid] = blk;
                s_meta[tid] = q < cnt ? s_lmeta[q] : 0;
                if (blk >= 0) {
                    s_bx[tid] = blk % g.nbx;
                    s_by[tid] = blk / g.nbx;
                }
                s_np[tid] = 0;
                s_nT[tid] = 0;
            }
            __syncthreads();
            // stage p and T of each block plus a 1-cell halo: both buffers beside the owner's parity,
            // selected afterwards, so the staging waits for one memory round trip instead of two
            for (int i = tid; i < K * TV; i += NT) {
                const int k = i / TV;
                if (s_blk[k] < 0) continue;
                const int j = i - k * TV;
                const int lx = j % E, ly = j / E;
                const int gx = wrapc(s_bx[k] * B + lx - 1, g.nx, g.bc);
                const int gy = wrapc(s_by[k] * B + ly - 1, g.ny, g.bc);
                const int ob = gx / B + g.nbx * (gy / B);
                const size_t gi = (size_t)gx + (size_t)g.nx * gy;
                const uint8_t pp = f.par_cur[ob], pT = f.par_cur[nb + ob];
                const R p0 = P.p[0][gi], p1 = P.p[1][gi], T0 = P.T[0][gi], T1 = P.T[1][gi];
                sp[i] = pp ? p1 : p0;
                sT[i] = pT ? T1 : T0;
            }
            __syncthreads();
#pragma unroll
            for (int c = 0; c < CPT; ++c) {
                const int k = (V >= NT) ? 0 : tid / V;
                const int v = (V >= NT) ? tid + c * NT : tid - k * V;
                const int blk = s_blk[k];
                if (blk < 0) continue;
                const int m = s_meta[k];
                const int lx = v % B, ly = v / B;
                const int ti = k * TV + (lx + 1) + SY * (ly + 1);
                const int bx = s_bx[k], by = s_by[k];
                const size_t gi = (size_t)(bx * B + lx) + (size_t)g.nx * (by * B + ly);
                const R pc = sp[ti], Tc = sT[ti];
                R pn = pc;
                if (m & 1) {   // Evolve_p (kernel.cu:220-241)
                    if constexpr (std::is_same<R, float>::value)
                        pn = den_p_f32<2>(pc, Tc, sp[ti + 1], sp[ti - 1], sp[ti + SY], sp[ti - SY], pc, pc, P.c32);
                    else
                        pn = den_p_new<R>(pc, Tc, sp[ti + 1], sp[ti - 1], sp[ti + SY], sp[ti - SY], pc, pc, f0, f1, f2, f3, dt, delta, eps2, gam);
                    ((m & 4) ? P.p[0] : P.p[1])[gi] = pn;
                    if (pn >= thr_p && pn <= thr_p_hi) s_np[k] = 1;
                    if (!isfinite(pn)) raise_status(f.status, 5);
                }
                if (m & 2) {   // Evolve_T (kernel.cu:286-289, :468-489)
                    R Tn;
                    if constexpr (std::is_same<R, float>::value)
                        Tn = den_T_f32<2, true>(Tc, sT[ti + 1], sT[ti - 1], sT[ti + SY], sT[ti - SY], Tc, Tc, (m & 1) != 0, pn, pc, P.c32);
                    else
                        Tn = den_T_new<R, true>(Tc, sT[ti + 1], sT[ti - 1], sT[ti + SY], sT[ti - SY], Tc, Tc, (m & 1) != 0, pn, pc, f1, dt);
                    ((m & 8) ? P.T[0] : P.T[1])[gi] = Tn;
                    if (fabs(Tn - Tc) >= thr_T) s_nT[k] = 1;
                    if (!isfinite(Tn)) raise_status(f.status, 5);
                }
            }
            __syncthreads();
            // wake-up tests and scatter: self + 6 faces per channel (kernel.cu:577-634), one
            // neighbour per thread (thread (2 k + ch) * 7 + n), from the block coordinates
            if (tid < K * 14) {
                const int k = tid / 14, r = tid - k * 14, ch = r / 7, n = r - ch * 7;
                const int blk = s_blk[k];
                if (blk >= 0 && ((s_meta[k] >> ch) & 1)) {
                    const int t = ch ? s_nT[k] : s_np[k];
                    if (n == 0) f.next[(size_t)ch * nb + blk] = (uint8_t)t;
                    if (t) {
                        const int nbk = block_nb_k(g, s_bx[k], s_by[k], 0, n);
                        if (nbk >= 0) f.wake_nxt[(size_t)ch * nb + nbk] = 1;
                    }
                }
            }
            __syncthreads();
        }
    }
}

}  // namespace dba

// k_dendrite3.cuh -- 3-D dendrite step, one CTA per tile of 32 x 8 x 8 cells: FP64, and FP32
// where the shape does not suit the queue-fed tiles of k_dendrite_tile.cuh.
//
// Same DBA semantics and point arithmetic as dendrite_step (k_dendrite.cuh), in one
// kernel: a CTA reads its tile's flags and ends when no block is active (about 2 ns per
// idle tile over the grid, so no list is built); otherwise
//   * p and T of the tile plus one cell are staged as 16-byte pieces, each inside one block
//     whose parity picks the buffer, and only in blocks that are active or share a face with
//     an active block of the tile;
//   * a thread owns a column of 8 cells and slides along z with the z neighbours in registers;
//     a warp holds 8 x 4 columns, one block of 8 or two of 4, so the warps of inactive blocks
//     skip the update, and with a 40-element pitch its four row segments fall on
//     distinct banks;
//   * a cell at a zero-flux wall is its own neighbour: its offset to that side is 0, so
//     nothing is staged beyond a wall.
// What bounds it: the latency of the flag, parity and staging round trips of a thin active
// shell (three to six resident CTAs per SM hide them for each other), then FP64 issue.
// The kernel before worked on one 4^3 block of 64 cells per quarter CTA and staged 216 cells
// for it, each with its own index arithmetic.
// Measured per step: 256^3 FP64 in 4^3 blocks, 16 % (p) and 44 % (T) of them active, 214 ->
// 84 us; 200 x 136 x 104 FP32 in 8^3 blocks, every block, 42.7 -> 22.2 us.
#pragma once

#include "k_common.cuh"
#include "k_dendrite.cuh"

namespace dba {

template <typename R, int B>
struct Den3 {
    static constexpr int NT = 256;
    static constexpr int TX = 32, TY = 8, TZ = 8;
    static constexpr int NBX = TX / B, NBY = TY / B, NBZ = TZ / B, NBT = NBX * NBY * NBZ;
    static constexpr int RX = NBX + 2, RY = NBY + 2, RZ = NBZ + 2, NR = RX * RY * RZ;
    static constexpr int PC = 16 / (int)sizeof(R);       // cells per staged piece
    static constexpr int SP = 40;                        // row pitch: column x at x + 4
    static constexpr int SH = TY + 2, SD = TZ + 2, PL = SP * SH, SV = PL * SD;
    static constexpr int NPR = TX / PC + 2;              // pieces per staged row: x from -PC to TX + PC - 1
    static constexpr int NPF = NPR * SH * SD;
    static constexpr size_t smem = sizeof(R) * 2 * SV;
    static constexpr int MINB = sizeof(R) == 8 ? 3 : 4;  // resident CTAs per SM
    static_assert(NBT <= 32 && TX % B == 0 && 8 % B == 0 && B % PC == 0 && 4 % PC == 0, "tile shape");
};

template <typename R, int B, bool DBA>
__global__ void __launch_bounds__(256, Den3<R, B>::MINB) dendrite3_step(GridP g, FlagP f, DenP<R> P)
{
    using S = Den3<R, B>;
    constexpr int NT = S::NT, SP = S::SP, PL = S::PL, SV = S::SV;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R* sp = reinterpret_cast<R*>(smem_raw);              // [SD][SH][SP]
    R* sT = sp + SV;
    __shared__ uint8_t s_tab[S::NR];                     // blocks around the tile: bit 0 p parity, 1 T parity, 2 staged
    __shared__ unsigned s_act[2], s_pq[2];               // the tile's blocks, p and T: active; parity
    __shared__ int s_hit[2][S::NBT];                     // wake tests
    const int tid = threadIdx.x, nb = g.nb;
    const int ntx = (g.nx + S::TX - 1) / S::TX, nty = (g.ny + S::TY - 1) / S::TY;
    const int tx = blockIdx.x % ntx, ty = (blockIdx.x / ntx) % nty, tz = blockIdx.x / (ntx * nty);
    const int X0 = tx * S::TX, Y0 = ty * S::TY, Z0 = tz * S::TZ;
    const int bx0 = X0 / B, by0 = Y0 / B, bz0 = Z0 / B;
    const int vx = min(S::TX, g.nx - X0), vy = min(S::TY, g.ny - Y0), vz = min(S::TZ, g.nz - Z0);

    if (tid < 32) {                                      // bookkeeping: the tile's blocks on one warp
        const int x = bx0 + tid % S::NBX, y = by0 + (tid / S::NBX) % S::NBY, z = bz0 + tid / (S::NBX * S::NBY);
        const bool valid = tid < S::NBT && x < g.nbx && y < g.nby && z < g.nbz;
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
            s_hit[0][tid] = 0;
            s_hit[1][tid] = 0;
        }
        count_stats(f.stats, act, valid);
        const unsigned m0 = __ballot_sync(0xffffffffu, act & 1), m1 = __ballot_sync(0xffffffffu, act & 2);
        const unsigned m2 = __ballot_sync(0xffffffffu, pp != 0), m3 = __ballot_sync(0xffffffffu, pT != 0);
        if (tid == 0) {
            s_act[0] = m0;
            s_act[1] = m1;
            s_pq[0] = m2;
            s_pq[1] = m3;
        }
    }
    __syncthreads();
    const unsigned ap = s_act[0], aT = s_act[1], any = ap | aT;
    if (any == 0) return;

    for (int r = tid; r < S::NR; r += NT) {
        const int rx = r % S::RX - 1, ry = (r / S::RX) % S::RY - 1, rz = r / (S::RX * S::RY) - 1;
        auto on = [&](int x, int y, int z) {             // active block (x, y, z) of the tile
            return x >= 0 && x < S::NBX && y >= 0 && y < S::NBY && z >= 0 && z < S::NBZ &&
                   ((any >> (x + S::NBX * (y + S::NBY * z))) & 1u);
        };
        unsigned v = 0;
        if (on(rx, ry, rz) || on(rx - 1, ry, rz) || on(rx + 1, ry, rz) || on(rx, ry - 1, rz) || on(rx, ry + 1, rz) ||
            on(rx, ry, rz - 1) || on(rx, ry, rz + 1)) {
            int x = bx0 + rx, y = by0 + ry, z = bz0 + rz;
            if (!g.bc) {
                x = wrap_p(x, g.nbx);
                y = wrap_p(y, g.nby);
                z = wrap_p(z, g.nbz);
            }
            // a block beyond a zero-flux wall, or past the grid's last tile, is not staged
            if (x >= 0 && x < g.nbx && y >= 0 && y < g.nby && z >= 0 && z < g.nbz) {
                const int b = x + g.nbx * (y + g.nby * z);
                v = 4u | (f.par_cur[b] ? 1u : 0u) | (f.par_cur[nb + b] ? 2u : 0u);
            }
        }
        s_tab[r] = (uint8_t)v;
    }
    __syncthreads();
    for (int i = tid; i < S::NPF; i += NT) {
        const int c = i % S::NPR, ry = (i / S::NPR) % S::SH, rz = i / (S::NPR * S::SH);
        const int lx = (c - 1) * S::PC, ly = ry - 1, lz = rz - 1;
        if (lx > vx || ly > vy || lz > vz) continue;
        const unsigned v = s_tab[(lx + B) / B + S::RX * ((ly + B) / B + S::RY * ((lz + B) / B))];
        if (!(v & 4u)) continue;
        // (a staged block is inside the grid, beyond its edge only where the grid is periodic)
        const int gx = wrap_p(X0 + lx, g.nx), gy = wrap_p(Y0 + ly, g.ny), gz = wrap_p(Z0 + lz, g.nz);
        const size_t gi = (size_t)gx + (size_t)g.nx * ((size_t)gy + (size_t)g.ny * gz);
        R* d = sp + rz * PL + ry * SP + lx + 4;
        cp_async16(d, ((v & 1u) ? P.p[1] : P.p[0]) + gi);
        cp_async16(d + SV, ((v & 2u) ? P.T[1] : P.T[0]) + gi);
    }
    cp_async_commit();
    cp_async_wait0();
    __syncthreads();

    const int w = tid >> 5, lane = tid & 31;
    const int cx = 8 * (w & 3) + (lane & 7), cy = 4 * (w >> 2) + (lane >> 3);
    const int kc = cx / B + S::NBX * (cy / B);           // the column's lowest block
    unsigned col = 0;                                    // the column's active blocks
#pragma unroll
    for (int j = 0; j < S::NBZ; ++j) col |= ((any >> (kc + j * S::NBX * S::NBY)) & 1u) << j;
    if (col) {
        const R f0 = (R)P.f0, f1 = (R)P.f1, f2 = (R)P.f2, f3 = (R)P.f3;
        const R dt = (R)P.dt, delta = (R)P.delta, eps2 = (R)P.eps2, gam = (R)P.gamma;
        const R thr_p = (R)P.thr_p, thr_p_hi = (R)P.thr_p_hi, thr_T = (R)P.thr_T;
        // neighbour offsets; 0 at a zero-flux wall
        const int dxm = g.bc && X0 + cx == 0 ? 0 : -1, dxp = g.bc && X0 + cx == g.nx - 1 ? 0 : 1;
        const int dym = g.bc && Y0 + cy == 0 ? 0 : -SP, dyp = g.bc && Y0 + cy == g.ny - 1 ? 0 : SP;
        int si = PL + (cy + 1) * SP + cx + 4;
        const int i0 = g.bc && Z0 == 0 ? si : si - PL;
        R pm = sp[i0], pc = sp[si], Tm = sT[i0], Tc = sT[si];
        const size_t nxy = (size_t)g.nx * g.ny;
        size_t gi = (size_t)(X0 + cx) + (size_t)g.nx * ((size_t)(Y0 + cy) + (size_t)g.ny * Z0);
        bool bad = false;
#pragma unroll
        for (int j = 0; j < S::NBZ; ++j) {
            const int k = kc + j * S::NBX * S::NBY;
            const bool pa = (ap >> k) & 1u, Ta = (aT >> k) & 1u;
            if (!(pa || Ta)) {                           // (a tile's last layers may lie outside the grid)
                si += B * PL;
                gi += B * nxy;
                if (j + 1 < S::NBZ) {
                    pm = sp[si - PL]; pc = sp[si]; Tm = sT[si - PL]; Tc = sT[si];
                }
                continue;
            }
            R* po = ((s_pq[0] >> k) & 1u) ? P.p[0] : P.p[1];
            R* to = ((s_pq[1] >> k) & 1u) ? P.T[0] : P.T[1];
            bool hp = false, hT = false;
#pragma unroll 2
            for (int z = 0; z < B; ++z) {
                const int iq = g.bc && Z0 + j * B + z == g.nz - 1 ? si : si + PL;
                const R pq = sp[iq], Tq = sT[iq];
                R pn = pc;
                if (pa) {                                // Evolve_p (kernel.cu:220-241)
                    if constexpr (sizeof(R) == 4)
                        pn = den_p_f32<3>(pc, Tc, sp[si + dxp], sp[si + dxm], sp[si + dyp], sp[si + dym], pq, pm, P.c32);
                    else
                        pn = den_p_new<R>(pc, Tc, sp[si + dxp], sp[si + dxm], sp[si + dyp], sp[si + dym], pq, pm, f0, f1,
                                          f2, f3, dt, delta, eps2, gam);
                    po[gi] = pn;
                    hp |= pn >= thr_p && pn <= thr_p_hi;
                    bad |= !isfinite(pn);
                }
                if (Ta) {                                // Evolve_T (kernel.cu:286-289, :468-489)
                    R Tn;
                    if constexpr (sizeof(R) == 4)
                        Tn = den_T_f32<3, DBA>(Tc, sT[si + dxp], sT[si + dxm], sT[si + dyp], sT[si + dym], Tq, Tm, pa, pn,
                                               pc, P.c32);
                    else
                        Tn = den_T_new<R, DBA>(Tc, sT[si + dxp], sT[si + dxm], sT[si + dyp], sT[si + dym], Tq, Tm, pa, pn,
                                               pc, f1, dt);
                    to[gi] = Tn;
                    hT |= fabs(Tn - Tc) >= thr_T;
                    bad |= !isfinite(Tn);
                }
                pm = pc; pc = pq; Tm = Tc; Tc = Tq;
                si += PL;
                gi += nxy;
            }
            if (DBA && hp) s_hit[0][k] = 1;
            if (DBA && hT) s_hit[1][k] = 1;
        }
        if (bad) raise_status(f.status, 5);
    }
    if (!DBA) return;
    __syncthreads();
    // wake-up tests and scatter: self + 6 faces per channel (kernel.cu:577-634), one neighbour per thread
    for (int i = tid; i < S::NBT * 14; i += NT) {
        const int k = i / 14, r = i - k * 14, ch = r / 7, n = r - ch * 7;
        if (!(((ch ? aT : ap) >> k) & 1u)) continue;
        const int x = bx0 + k % S::NBX, y = by0 + (k / S::NBX) % S::NBY, z = bz0 + k / (S::NBX * S::NBY);
        const int hit = s_hit[ch][k];
        if (n == 0) f.next[(size_t)ch * nb + x + g.nbx * (y + g.nby * z)] = (uint8_t)hit;
        if (hit) {
            const int nbk = block_nb_k(g, x, y, z, n);
            if (nbk >= 0) f.wake_nxt[(size_t)ch * nb + nbk] = 1;
        }
    }
}

}  // namespace dba

// k_modelb.cuh -- one step of the reactive Model B (ternary Flory-Huggins
// Cahn-Hilliard + reaction) over the active blocks: FP64, and FP32 in 3-D
// (reference: example_Reactive_ModelB/kernel.cu and Conserved/kernel.cu).
//
// Reference per DBA step: Calc_mu_wakeup (:519) writes b, the chemical
// potentials dfdx/dfdy/dfdz (27-point Laplacians, logs) and metric = |lap z|
// for active blocks; Update_wakeup (:594) advances x, y, z with 27-point
// Laplacians of the potentials and the exp reaction term, reading potentials
// of inactive neighbour blocks as they were at those blocks' last active step;
// Swap_wakeup (:469) commits; Wakeup_Next (:657) tests metric > Metric_eps;
// Wakeup_Neighbor (:716) wakes the 6 face neighbours.
//
// Two kernels, one CTA per tile of 1024 to 2048 cells (3-D) or 32 x 8..32 cells (2-D),
// in each of which a tile without an active block ends after reading its flags:
//
//   modelb_mu      stages x, y, z of the tile and a 1-cell halo in shared memory (16-byte
//                  pieces, each inside one block, whose parity picks the buffer), writes
//                  the potentials of the active blocks to the potential arrays, and does
//                  the step's block bookkeeping: parity flip, flag clearing, wake-up
//                  tests and scatter;
//   modelb_update  stages the potentials (one buffer, hence no parity) -- an active block's
//                  are this step's, an inactive one's those of its last active step, as
//                  in the reference -- and writes x, y, z to the active blocks' other
//                  ping-pong buffers.
//
// What bounds it: FP64 issue.  The 27-point Laplacians are kept in the reference's term
// order, so no partial sum is shared between cells: about 270 FP64 operations per cell
// in modelb_mu and 155 in modelb_update.  Storing the potentials once costs 48 bytes per
// cell of traffic and computes each once; a single kernel that recomputed them on every
// block's halo (the form before) did 3.4 times the potential work at 4^3 blocks and
// staged 8 cells for each that it advanced.
// A thread owns 4 cells along z (8 in FP32 8^3 blocks) and walks down the planes, one field
// after the other; a cell's sums take each plane's values as it arrives (LapZ), so a value
// is loaded 9 to 14 times, not 27, and 16 registers carry what a window of three planes
// would need 54 for.  The pointwise part is one copy of the code per kernel (unrolled
// over the cells, its logarithms and exponentials overflowed the instruction cache), and
// 64 registers leave four CTAs per SM: 3 CTAs at 80 registers took 792 us where 4 take 708.
// Measured per step, every block active, before -> now: 256^3 FP64 in 4^3 blocks 5167 ->
// 708 us, 192^3 FP32 in 8^3 blocks (regular) 554 -> 168 us, 4^3 blocks 1088 -> 187 us;
// 768^2 FP64 in 4^2 blocks 72.7 -> 29.0 us, conserved in 16^2 blocks 67.5 -> 47.9 us.  A 2-D grid of
// many tiles that is nearly all asleep was faster one block at a time (idle CTAs of two
// kernels): 1024^2 in 4^2 blocks 2 % active 10.1 -> 11.8, 12 % 20.5 -> 19.0, 43 % 62 -> 33.
// The Nz == 1 form keeps the reference's 27-term sum with the z neighbours
// wrapped onto the cell itself.
#pragma once

#include "fpmath.h"
#include "k_common.cuh"

namespace dba {

template <typename R>
struct MBP {
    R* x[2];
    R* y[2];
    R* z[2];
    R* mu[3];                       // persisted potentials (x, y, z)
    double inv_dx2;                 // 1.0 / (dx * dx)
    double c0x, c0y, c0z;           // -1.0 + 1.0/r{x,y,z}
    double rx, ry, rz;
    double chi_xy, chi_xz, chi_yz, chi_xb, chi_yb, chi_zb;
    double ex, ey, ez;
    double phi_term;                // p_gel*phi*phi/2/(1-z_crit) with phi = 0
    double logK_rz;                 // log(K)/rz
    double nvx, mvy, dvz;           // n*vx, m*vy, vz
    double dtvx, dtvy, dtvz;        // dt*vx, dt*vy, dt*vz
    double dn, dm;                  // n, m
    double Mx, My, Mz, k0;
    double thr;                     // Metric_eps
    int conserved;
    // 1 / r{x,y,z} where that is exact (a power of two: the product then rounds as the
    // quotient does), else 0: divide
    double irx, iry, irz;
};

template <typename R> __device__ __forceinline__ R log_r(R v);
template <> __device__ __forceinline__ double log_r<double>(double v) { return dba_log(v); }
template <> __device__ __forceinline__ float log_r<float>(float v) { return logf(v); }
template <typename R> __device__ __forceinline__ R exp_r(R v);
template <> __device__ __forceinline__ double exp_r<double>(double v) { return dba_exp(v); }
template <> __device__ __forceinline__ float exp_r<float>(float v) { return expf(v); }

// 27-point isotropic Laplacian of a cell from the 3 x 3 values v of the planes z + 1, z,
// z - 1, fed in that order: value 3 (dy + 1) + dx + 1 of a plane.  FP64 adds the
// reference's terms in its order (kernel.cu:332-344): faces +x -x +y -y +z -z, the 12
// edges plane z first, then z + 1, z - 1, the 8 corners z + 1 first.  FP32 sums each
// plane's faces and diagonals first: 14 sums instead of 26, and an error no larger.
template <typename R>
struct LapZ {
    R c, F, E, C, e5, e7, e1, e3;      // centre; sums of faces, edges, corners; plane z + 1's values until plane z is in
    __device__ __forceinline__ void above(const R* p)
    {
        if constexpr (sizeof(R) == 8) {
            C = p[8] + p[6] + p[0] + p[2];
            F = p[4];
            e5 = p[5]; e7 = p[7]; e1 = p[1]; e3 = p[3];
        } else {
            F = p[4];
            E = (p[5] + p[3]) + (p[7] + p[1]);
            C = (p[8] + p[0]) + (p[6] + p[2]);
        }
    }
    __device__ __forceinline__ void centre(const R* o)
    {
        c = o[4];
        if constexpr (sizeof(R) == 8) {
            F = o[5] + o[3] + o[7] + o[1] + F;
            E = o[8] + o[2] + o[6] + o[0] + e5 + e7 + e1 + e3;
        } else {
            F = F + ((o[5] + o[3]) + (o[7] + o[1]));
            E = E + ((o[8] + o[0]) + (o[6] + o[2]));
        }
    }
    __device__ __forceinline__ R below(const R* m, R inv_dx2)
    {
        if constexpr (sizeof(R) == 8) {
            F = F + m[4];
            E = E + m[5] + m[7] + m[1] + m[3];
            C = C + m[8] + m[6] + m[0] + m[2];
        } else {
            F = F + m[4];
            E = E + ((m[5] + m[3]) + (m[7] + m[1]));
            C = C + ((m[8] + m[0]) + (m[6] + m[2]));
        }
        return inv_dx2 * ((R)(-64.0 / 15.0) * c + (R)(7.0 / 15.0) * F + (R)0.1 * E + (R)(1.0 / 30.0) * C);
    }
};

// Tile shapes: 3-D 32 x 8 x 4 (4^3 blocks), 16 x 8 x 8 (8^3, FP64), 32 x 8 x 8 (8^3, FP32):
// a tile holds whole blocks, and the staged box of three fields leaves room for 4 CTAs of
// 256 threads (modelb_mu at 32 x 8 x 8 in FP64: 86 KB, 2 CTAs, and half the speed; FP32 8^3
// with 4 cells per thread and CTAs of 512: 223 us where 8 cells and 256 threads take 168).
// 2-D: 32 x 8 (4^2, 8^2 blocks), TALL 32 x 16 (mb_tall), 32 x 16 or 32 x 32 (16^2, 32^2 blocks).
template <typename R, int D, int B, bool TALL = false>
struct MBShape {
    static constexpr int TX = D == 3 && B == 8 && sizeof(R) == 8 ? 16 : 32;
    static constexpr int TY = D == 3 ? 8 : (B > 8 ? B : (TALL ? 16 : 8)), TZ = D == 3 ? B : 1;   // tile in cells
    static constexpr int NBX = TX / B, NBY = TY / B, NBZ = D == 3 ? TZ / B : 1, NBT = NBX * NBY * NBZ;
    static constexpr int RX = NBX + 2, RY = NBY + 2, RZ = D == 3 ? NBZ + 2 : 1, NR = RX * RY * RZ;
    static constexpr int PC = 16 / (int)sizeof(R);       // cells per staged piece (B is a multiple)
    static constexpr int SW = TX + 2 * PC, SH = TY + 2, SD = D == 3 ? TZ + 2 : 1;           // staged box
    static constexpr int PL = SW * SH, SV = PL * SD;     // one staged plane, one staged field
    static constexpr int NPR = SW / PC;                  // pieces per staged row
    static constexpr int NC = D == 3 ? (sizeof(R) == 4 ? B : 4) : TY / 8;       // cells per thread: along z, in 2-D along y
    static constexpr int CELLS = TX * TY * TZ, NT = CELLS / NC;
    static constexpr int MINB = 1024 / NT;               // resident CTAs per SM: 64 registers per thread
    static constexpr size_t smem_mu = sizeof(R) * 3 * SV;
    static constexpr size_t smem_chg = sizeof(double) * 3 * CELLS;      // modelb_update, conserved: the cells' changes,
    static constexpr size_t smem_cons = smem_mu > smem_chg ? smem_mu : smem_chg;   // in the staged potentials' place
    static_assert(NBT <= 32 && NBT >= 1 && B % PC == 0 && TX % B == 0 && TY % B == 0, "a tile's blocks fit one warp");
    static_assert(NT == 256 && B % NC == 0, "a thread's cells lie in one block");
    // first cell (x, y, z) of thread tid
    static __device__ __forceinline__ void first(int tid, int& x, int& y, int& z)
    {
        x = tid % TX;
        if (D == 3) {
            y = (tid / TX) % TY;
            z = NC * (tid / (TX * TY));
        } else {
            y = NC * (tid / TX);
            z = 0;
        }
    }
};

// The tile of a CTA: first cell, first block, and the part of it inside the grid (a grid
// whose edges are multiples of the block edge only ends inside its last tiles).
template <typename S, int D, int B>
struct MBTileAt {
    int X0, Y0, Z0, bx, by, bz, vx, vy, vz;
    __device__ __forceinline__ MBTileAt(const GridP& g)
    {
        const int ntx = (g.nx + S::TX - 1) / S::TX, nty = (g.ny + S::TY - 1) / S::TY;
        const int t = blockIdx.x, tx = t % ntx, ty = (t / ntx) % nty, tz = t / (ntx * nty);
        X0 = tx * S::TX; Y0 = ty * S::TY; Z0 = D == 3 ? tz * S::TZ : 0;
        bx = X0 / B; by = Y0 / B; bz = D == 3 ? Z0 / B : 0;
        vx = min(S::TX, g.nx - X0); vy = min(S::TY, g.ny - Y0); vz = D == 3 ? min(S::TZ, g.nz - Z0) : 1;
    }
    // global id of the tile's block k, -1 outside the grid
    __device__ __forceinline__ int block(const GridP& g, int k) const
    {
        const int x = bx + k % S::NBX, y = by + (k / S::NBX) % S::NBY, z = bz + k / (S::NBX * S::NBY);
        return x < g.nbx && y < g.nby && z < g.nbz ? x + g.nbx * (y + g.nby * z) : -1;
    }
};

// Per-block FP64 sums of one value per cell of the tile (s_val[cell], cell = x + TX (y +
// TY z)), in the fixed order of block_tree_sums: runs of 32 consecutive cells of a block
// with strides 16..1, then the run sums.  One warp per block; blocks not in `mask` skipped.
template <typename S, int D, int B>
__device__ __forceinline__ void tile_block_sums(const double* s_val, unsigned mask, double* s_out)
{
    constexpr int V = ipow(B, D), SEG = V < 32 ? V : 32, RUNS = V / 32;
    const int lane = threadIdx.x & 31;
    for (int k = threadIdx.x >> 5; k < S::NBT; k += S::NT / 32) {
        if (!((mask >> k) & 1u)) continue;
        const int x0 = (k % S::NBX) * B, y0 = ((k / S::NBX) % S::NBY) * B, z0 = (k / (S::NBX * S::NBY)) * B;
        auto cell = [&](int v) {
            return s_val[x0 + v % B + S::TX * (y0 + (v / B) % B + S::TY * (z0 + (D == 3 ? v / (B * B) : 0)))];
        };
        double out;
        if constexpr (V < 32) {
            double v = lane < V ? cell(lane) : 0.0;
#pragma unroll
            for (int h = SEG / 2; h >= 1; h /= 2) v += __shfl_down_sync(0xffffffffu, v, h, SEG);
            out = v;
        } else {
            double rs = 0.0;
            for (int r = 0; r < RUNS; ++r) {
                double v = cell(r * 32 + lane);
#pragma unroll
                for (int h = 16; h >= 1; h /= 2) v += __shfl_down_sync(0xffffffffu, v, h);
                v = __shfl_sync(0xffffffffu, v, 0);
                if (lane == r) rs = v;
            }
            if (RUNS > 1) {
#pragma unroll
                for (int h = (RUNS > 32 ? 16 : RUNS / 2); h >= 1; h /= 2) rs += __shfl_down_sync(0xffffffffu, rs, h);
            }
            out = rs;
        }
        if (lane == 0) s_out[k] = out;
    }
}

// The 16-byte pieces of the tile's part inside the grid and one cell around it: a thread
// keeps one piece of a plane (so its column, row and wrap are worked out once) and steps
// over the planes.  body(cell index, staged offset, index in the table of blocks).
template <typename S, int D, int B, typename T, typename F>
__device__ __forceinline__ void stage_pieces(const GridP& g, const T& t, F&& body)
{
    constexpr int PP = S::NPR * S::SH, ZP = PP <= S::NT ? S::NT / PP : 1;   // pieces of a plane; planes at once
    const int ph = PP <= S::NT ? (int)threadIdx.x / PP : 0;
    if (ph >= ZP) return;
    for (int i = (int)threadIdx.x - ph * PP; i < PP; i += PP <= S::NT ? PP : S::NT) {
        const int c = i % S::NPR, ry = i / S::NPR;
        const int lx = (c - 1) * S::PC, ly = ry - 1;
        if (lx > t.vx || ly > t.vy) continue;
        const int reg = (lx + B) / B + S::RX * ((ly + B) / B);
        const size_t row = (size_t)wrap_p(t.X0 + lx, g.nx) + (size_t)g.nx * wrap_p(t.Y0 + ly, g.ny);
        if constexpr (D == 3) {
            const size_t nxy = (size_t)g.nx * g.ny;
#pragma unroll 2
            for (int rz = ph; rz < S::SD && rz - 1 <= t.vz; rz += ZP)
                body(row + nxy * wrap_p(t.Z0 + rz - 1, g.nz), rz * S::PL + i * S::PC, reg + S::RX * S::RY * ((rz - 1 + B) / B));
        } else {
            body(row, i * S::PC, reg);
        }
    }
    cp_async_commit();
}

// Laplacians of a thread's NC cells from a staged field; s = the thread's first cell
template <typename S, typename R, int D>
__device__ __forceinline__ void column_laps(const R* s, R inv_dx2, R* lap)
{
    constexpr int NC = S::NC, SW = S::SW, PL = S::PL;
    auto load = [&](R* v, const R* at) {
#pragma unroll
        for (int j = 0; j < 9; ++j) v[j] = at[(j / 3 - 1) * SW + j % 3 - 1];
    };
    R v[9];
    if constexpr (D == 3) {
        LapZ<R> l[3];                                    // cells c, c + 1, c + 2 in turn
#pragma unroll
        for (int c = NC; c >= -1; --c) {                 // plane c: below c + 1, centre of c, above c - 1
            load(v, s + c * PL);
            if (c + 1 < NC) lap[c + 1] = l[(c + 1) % 3].below(v, inv_dx2);
            if (c >= 0 && c < NC) l[c % 3].centre(v);
            if (c >= 1) l[(c - 1) % 3].above(v);
        }
    } else {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            LapZ<R> l;
            load(v, s + c * SW);
            l.above(v);
            l.centre(v);
            lap[c] = l.below(v, inv_dx2);
        }
    }
}

template <typename R, int D, int B, bool DBA, bool TALL>
__global__ void __launch_bounds__((MBShape<R, D, B, TALL>::NT), (MBShape<R, D, B, TALL>::MINB)) modelb_mu(GridP g, FlagP f, MBP<R> P)
{
    using S = MBShape<R, D, B, TALL>;
    constexpr int NC = S::NC, SW = S::SW, PL = S::PL, SV = S::SV, NT = S::NT;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R* stage = reinterpret_cast<R*>(smem_raw);           // [x, y, z][SD][SH][SW]
    __shared__ uint8_t s_tab[S::NR];                     // blocks around the tile: buffer parity
    __shared__ unsigned s_fresh, s_own;                  // the tile's blocks: potentials computed; owned and active
    __shared__ int s_nx[S::NBT];
    const int tid = threadIdx.x;
    const MBTileAt<S, D, B> t(g);
    const int nb = g.nb;
    grid_wait();                                         // the step before

    if (tid < 32) {                                      // bookkeeping: the tile's blocks on one warp
        const int b = tid < S::NBT ? t.block(g, tid) : -1;
        int flagged = 0, act = 0, pp = 0;
        if (b >= 0) {
            pp = f.par_cur[b];
            flagged = DBA ? (f.wake_cur[b] ? 1 : 0) : 1;
            const int by = t.by + (tid / S::NBX) % S::NBY;
            act = (by >= g.ob0 && by < g.ob1) ? flagged : 0;
            f.wake_clr[b] = 0;
            if (!DBA) f.wake_nxt[b] = 1;
            f.par_nxt[b] = (uint8_t)(pp ^ act);
            if (P.conserved && !act) {
                f.bsum[b] = 0.0;
                f.bsum[nb + b] = 0.0;
                f.bsum[2 * nb + b] = 0.0;
            }
            s_nx[tid] = 0;
        }
        count_stats(f.stats, act, b >= 0);
        const unsigned mf = __ballot_sync(0xffffffffu, flagged != 0), mo = __ballot_sync(0xffffffffu, act != 0);
        if (tid == 0) {
            s_fresh = mf;
            s_own = mo;
        }
    }
    for (int r = tid; r < S::NR; r += NT) {
        int x = t.bx + r % S::RX - 1, y = t.by + (r / S::RX) % S::RY - 1, z = D == 3 ? t.bz + r / (S::RX * S::RY) - 1 : 0;
        x = wrap_p(x, g.nbx); y = wrap_p(y, g.nby);
        if (D == 3) z = wrap_p(z, g.nbz);
        // past the grid's last tiles there are entries that no staged piece refers to
        s_tab[r] = (x < g.nbx && y < g.nby && z < g.nbz) ? f.par_cur[x + g.nbx * (y + g.nby * z)] : (uint8_t)0;
    }
    __syncthreads();
    const unsigned fresh = s_fresh, own = s_own;
    if (fresh == 0) return;

    stage_pieces<S, D, B>(g, t, [&](size_t gi, int so, int reg) {
        const int par = s_tab[reg];
        cp_async16(stage + so, (par ? P.x[1] : P.x[0]) + gi);
        cp_async16(stage + SV + so, (par ? P.y[1] : P.y[0]) + gi);
        cp_async16(stage + 2 * SV + so, (par ? P.z[1] : P.z[0]) + gi);
    });
    cp_async_wait0();
    __syncthreads();

    const R inv_dx2 = (R)P.inv_dx2;
    int cx, cy, cz;
    S::first(tid, cx, cy, cz);
    const R* s0 = stage + (cy + 1) * SW + cx + S::PC + (D == 3 ? (cz + 1) * PL : 0);
    const int k = cx / B + S::NBX * (cy / B + S::NBY * (cz / B));   // the thread's block
    if ((fresh >> k) & 1u) {
        R lap[3][NC];
#pragma unroll
        for (int q = 0; q < 3; ++q) column_laps<S, R, D>(s0 + q * SV, inv_dx2, lap[q]);
        // potentials (Calc_mu, kernel.cu:371-388)
        auto over = [](R v, double r, double ir) { return ir != 0.0 ? v * (R)ir : v / (R)r; };
        bool hit = false;
        const size_t g0 = (size_t)(t.X0 + cx) + (size_t)g.nx * ((size_t)(t.Y0 + cy) + (size_t)g.ny * (t.Z0 + cz));
        // one copy of the code (4 logarithms a cell): the Laplacians shift down instead
#pragma unroll 1
        for (int c = 0; c < NC; ++c) {
            const R* s = s0 + c * (D == 3 ? PL : SW);
            const R X = s[0], Y = s[SV], Z = s[2 * SV];
            const R lapx = lap[0][0], lapy = lap[1][0], lapz = lap[2][0];
#pragma unroll
            for (int q = 0; q < 3; ++q)
#pragma unroll
                for (int j = 0; j + 1 < NC; ++j) lap[q][j] = lap[q][j + 1];
            const R bb = (R)1.0 - X - Y - Z;
            const R lb = log_r<R>(bb);
            const R ux = (R)P.c0x + (R)P.chi_xy * Y + (R)P.chi_xz * Z + (R)P.chi_xb * bb - (R)P.chi_xb * X -
                         (R)P.chi_yb * Y - (R)P.chi_zb * Z + over(log_r<R>(X), P.rx, P.irx) - lb - (R)P.ex * lapx;
            const R uy = (R)P.c0y + (R)P.chi_xy * X + (R)P.chi_yz * Z + (R)P.chi_yb * bb - (R)P.chi_xb * X -
                         (R)P.chi_yb * Y - (R)P.chi_zb * Z + over(log_r<R>(Y), P.ry, P.iry) - lb - (R)P.ey * lapy;
            const R uz = (R)P.c0z + (R)P.chi_xz * X + (R)P.chi_yz * Y + (R)P.chi_zb * bb - (R)P.chi_xb * X -
                         (R)P.chi_yb * Y - (R)P.chi_zb * Z + over(log_r<R>(Z), P.rz, P.irz) - lb - (R)P.phi_term -
                         (R)P.ez * lapz - (R)P.logK_rz;
            const size_t gi = g0 + c * (size_t)g.nx * (D == 3 ? g.ny : 1);
            P.mu[0][gi] = ux;
            P.mu[1][gi] = uy;
            P.mu[2][gi] = uz;
            hit |= fabs(lapz) > (R)P.thr;                    // Wakeup_Next :697
        }
        if (DBA && hit) s_nx[k] = 1;
    }
    if (!DBA) return;
    __syncthreads();
    // the own active blocks' tests, and the scatter to self and 6 faces, one neighbour per thread
    for (int i = tid; i < S::NBT * 7; i += NT) {
        const int k = i / 7, n = i - 7 * k;
        if (!((own >> k) & 1u)) continue;
        if (n == 0) f.next[t.block(g, k)] = (uint8_t)s_nx[k];
        if (s_nx[k]) {
            const int nbk = block_nb_k(g, t.bx + k % S::NBX, t.by + (k / S::NBX) % S::NBY, t.bz + k / (S::NBX * S::NBY), n);
            if (nbk >= 0) f.wake_nxt[nbk] = 1;
        }
    }
}

template <typename R, int D, int B, bool DBA, bool TALL>
__global__ void __launch_bounds__((MBShape<R, D, B, TALL>::NT), (MBShape<R, D, B, TALL>::MINB)) modelb_update(GridP g, FlagP f, MBP<R> P)
{
    using S = MBShape<R, D, B, TALL>;
    constexpr int NC = S::NC, SW = S::SW, PL = S::PL, SV = S::SV;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R* stage = reinterpret_cast<R*>(smem_raw);           // [x, y, z potentials][SD][SH][SW]
    __shared__ unsigned s_own, s_par;
    __shared__ double s_bsum[3][S::NBT];
    const int tid = threadIdx.x;
    const MBTileAt<S, D, B> t(g);
    grid_wait();                                         // modelb_mu
    if (tid < 32) {
        const int b = tid < S::NBT ? t.block(g, tid) : -1;
        int act = 0, pp = 0;
        if (b >= 0) {
            const int by = t.by + (tid / S::NBX) % S::NBY;
            act = (by >= g.ob0 && by < g.ob1) ? (DBA ? (f.wake_cur[b] ? 1 : 0) : 1) : 0;
            pp = f.par_cur[b];
        }
        const unsigned mo = __ballot_sync(0xffffffffu, act != 0), mp = __ballot_sync(0xffffffffu, pp != 0);
        if (tid == 0) {
            s_own = mo;
            s_par = mp;
        }
    }
    __syncthreads();
    const unsigned own = s_own, par = s_par;
    if (own == 0) return;

    stage_pieces<S, D, B>(g, t, [&](size_t gi, int so, int) {
#pragma unroll
        for (int q = 0; q < 3; ++q) cp_async16(stage + q * SV + so, P.mu[q] + gi);
    });

    const R inv_dx2 = (R)P.inv_dx2;
    int cx, cy, cz;
    S::first(tid, cx, cy, cz);
    const R* s0 = stage + (cy + 1) * SW + cx + S::PC + (D == 3 ? (cz + 1) * PL : 0);
    const int k = cx / B + S::NBX * (cy / B + S::NBY * (cz / B));   // the thread's block
    const bool on = (own >> k) & 1u;
    const size_t g0 = (size_t)(t.X0 + cx) + (size_t)g.nx * ((size_t)(t.Y0 + cy) + (size_t)g.ny * (t.Z0 + cz));
    const size_t gs = (size_t)g.nx * (D == 3 ? g.ny : 1);
    const int src = (par >> k) & 1u;
    cp_async_wait0();
    __syncthreads();
    R lap[3][NC];                                        // Laplacians, then (conserved) the changes
    if (on) {
#pragma unroll
        for (int q = 0; q < 3; ++q) column_laps<S, R, D>(s0 + q * SV, inv_dx2, lap[q]);
        // update (Update, kernel.cu:419-434; Conserved/kernel.cu:428-440); one copy of the code:
        // the Laplacians shift down and the changes follow them
#pragma unroll 1
        for (int c = 0; c < NC; ++c) {
            const R* sc = s0 + c * (D == 3 ? PL : SW);
            const R mx = sc[0], my = sc[SV], mz = sc[2 * SV];
            const size_t gi = g0 + c * gs;
            const R X = (src ? P.x[1] : P.x[0])[gi], Y = (src ? P.y[1] : P.y[0])[gi], Z = (src ? P.z[1] : P.z[0])[gi];
            const R Rr = (R)P.k0 * (exp_r<R>((R)P.nvx * mx + (R)P.mvy * my) - exp_r<R>((R)P.dvz * mz));
            const R chx = (R)P.dtvx * ((R)P.Mx * lap[0][0] - (R)P.dn * Rr);
            const R chy = (R)P.dtvy * ((R)P.My * lap[1][0] - (R)P.dm * Rr);
            const R chz = (R)P.dtvz * ((R)P.Mz * lap[2][0] + Rr);
            const R xn = X + chx, yn = Y + chy, zn = Z + chz;
            (src ? P.x[0] : P.x[1])[gi] = xn;
            (src ? P.y[0] : P.y[1])[gi] = yn;
            (src ? P.z[0] : P.z[1])[gi] = zn;
            if (!isfinite(xn) || !isfinite(yn) || !isfinite(zn)) raise_status(f.status, 5);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
#pragma unroll
                for (int j = 0; j + 1 < NC; ++j) lap[q][j] = lap[q][j + 1];
                lap[q][NC - 1] = q == 0 ? chx : (q == 1 ? chy : chz);
            }
        }
    }
    if (!P.conserved) return;
    // per-block change sums in the fixed tree order
    __syncthreads();                                     // the staged potentials have been read
    double* s_chg = reinterpret_cast<double*>(smem_raw); // [x, y, z][CELLS]
    if (on) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int q = 0; q < 3; ++q)
                s_chg[q * S::CELLS + cx + S::TX * (D == 3 ? cy + S::TY * (cz + c) : cy + c)] = (double)lap[q][c];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 3; ++q) tile_block_sums<S, D, B>(s_chg + q * S::CELLS, own, s_bsum[q]);
    __syncthreads();
    if (tid < 3 * S::NBT) {
        const int q = tid / S::NBT, k = tid - q * S::NBT;
        if ((own >> k) & 1u) f.bsum[(size_t)q * g.nb + t.block(g, k)] = s_bsum[q][k];
    }
}

}  // namespace dba

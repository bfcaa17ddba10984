// k_kh_strip.cuh -- FP32 KH step of fully active regions: a warp marches down a strip.
//
// Same semantics and point formulas as kh_tile_step (k_kh_tile.cuh), for the tiles whose
// blocks and all blocks around them are active this step ("full" tiles; every tile in
// regular mode).  There nothing stale is read, so a step needs no staged neighbourhood:
// a warp takes 64 columns, two per lane (60 of them its own), and walks down 16 or 32 rows.
// A lane keeps the primitives of two rows, the face state, fluxes and flux difference of the
// row before; x neighbours come by shuffles (20 a row for 60 cells), y neighbours are
// registers; no shared memory, no barrier; the arithmetic is two-lane FP32 (k_pair.cuh).
// Tiles that are not full go to kh_tile_step.
//
//   kh_strip_scan    the bookkeeping of kh_tile_scan, and per tile: full, or listed; persists
//                    what the neighbours of a block that fell asleep since the step before can read
//                    stale, computed again from the buffers that step read
//   kh_strip_step    full tiles; per block: the largest signal speed (CFL), the wake-up test with its
//                    scatter
//   kh_tile_step     (DBA) the listed tiles, beside the strips (grid_release)
//
// What bounds it: latency at four warps per scheduler (128 registers), then instruction issue.
// The tile kernel spends 686 warp instructions on 32 cells: it computes primitives on 400,
// gradients on 320 and fluxes on 288 cells for 256, and moves every intermediate through
// shared memory (71 % of that pipe's peak).  One column per lane took 368 instructions on
// 28 cells and 75 us per regular 2048^2 step, this form 472 on 60 cells and 66.
// Measured per step, every block active, tile kernel -> this: 2048^2 DBA with the CFL step 120 ->
// 69 us, regular 114 -> 66; 4096^2 DBA 449 -> 246; 1024^2 DBA 36.9 -> 30.7, regular 35.5 -> 23.4.
// A DBA step's three kernels are launched beside one another (grid_release, grid_wait): the scan
// starts while the last tiles of the step before end, the strips' CTAs while it runs, and the
// tiles take the places that strips leave.  In plain order a step that uses no strips took 2 to 5 us
// more than tiles alone; now -0.7 to +0.9.
#pragma once

#include "k_common.cuh"
#include "k_kh.cuh"
#include "k_kh_tile.cuh"
#include "k_pair.cuh"

namespace dba {

struct KHStrip {
    static constexpr int OUT = 60;                       // columns a warp advances: two per lane, lanes 1 .. 30
    // independent warps, 16 per SM at 128 registers; DBA steps in one CTA per SM
    static constexpr int NT = 128, NTD = 512;
    // Rows a warp walks (a multiple of 16): 32, or 16 where 32 would leave most of the 148 x 16
    // resident warps idle.  us per regular step, 32 / 16 rows: 2048^2 (2240 warps at 32) 66 / 69,
    // 1024^2 (576) 47 / 35.
    static int rows(int nx, int ny) { return (long long)((nx + OUT - 1) / OUT) * (ny / 32) >= 2000 ? 32 : 16; }
};

// full[tile]: every block of the 16^2 tile and around it is active in the step last scanned, which took
// the tile by strips.  Counts of such tiles (whatever took them): of the step before, of this one,
// and the word that the next step counts into.
struct KHStripP {
    uint8_t* full = nullptr;
    const unsigned* cnt_prev = nullptr;
    unsigned *cnt_cur = nullptr, *cnt_next = nullptr;
    unsigned* taken = nullptr;                           // units taken beyond every warp's first
};

// Whether this step uses the strips: by the full tiles of the step before (either way the results
// are the same, bit for bit).  A warp walks its unit when any tile of it is full, so scattered
// quiet spots leave the strips' time as it is, while the tiles that are not full come on top.
// us per step, tiles / strips, at shares of full tiles (a quiet band; 4 quiet spots; 64):
//   1024^2 (4096 tiles)  92 % 36.8 / 35.6; 90 % 36.3 / 36.3; 86 % 36.1 / 37.1; 83 % 34.5 / 35.5; 76 % 33.9 / 37.2
//   1536^2               92 % 69.6 / 46.0; 72 % 57.1 / 39.0; 66 % 56.9 / 47.8; 64 % 71 / 60
//   2048^2 (16384 tiles) 92 % 114 / 74; 74 % 98.9 / 76.2; 64 % 89 / 75; 60 % 103 / 98; 55 % 79.6 / 74.3;
//                        45 % 69.7 / 71.5
// (A restored state starts with a count of all ones: strips on.)
__device__ __forceinline__ bool kh_strips_on(const GridP& g, const unsigned* cnt)
{
    const unsigned n = (unsigned)((g.nx / 16) * (g.ny / 16)), lacking = n - min(*cnt, n);
    return lacking <= (n >= 8192u ? 2u * n / 5u : n / 10u);   // 8192 tiles: 2^21 cells
}

// one cell's four quantities, and the formulas on them (the blocks that may fall asleep)
struct Row4 {
    float a, b, c, d;
};
__device__ __forceinline__ Row4 kh_row_grad(const Row4& p, const Row4& m, float h)
{
    return Row4{kh_grad<float>(p.a, m.a, h), kh_grad<float>(p.b, m.b, h), kh_grad<float>(p.c, m.c, h), kh_grad<float>(p.d, m.d, h)};
}
// x-face flux between a cell (w0, x gradients g0) and the one on its right, as Mass, Energy, Momx, Momy
__device__ __forceinline__ Row4 kh_row_fx(const KHK<float>& K, const Row4& w0, const Row4& g0, const Row4& w1, const Row4& g1)
{
    Row4 r;
    kh_getflux<float>(K, kh_face_m<float>(w1.a, g1.a, K.ex), kh_face_p<float>(w0.a, g0.a, K.ex), kh_face_m<float>(w1.b, g1.b, K.ex),
                      kh_face_p<float>(w0.b, g0.b, K.ex), kh_face_m<float>(w1.c, g1.c, K.ex), kh_face_p<float>(w0.c, g0.c, K.ex),
                      kh_face_m<float>(w1.d, g1.d, K.ex), kh_face_p<float>(w0.d, g0.d, K.ex), r.a, r.b, r.c, r.d);
    return r;
}
// y-face flux between a cell (w0, y gradients g0) and the one above it
__device__ __forceinline__ Row4 kh_row_fy(const KHK<float>& K, const Row4& w0, const Row4& g0, const Row4& w1, const Row4& g1)
{
    Row4 r;
    kh_getflux<float>(K, kh_face_m<float>(w1.a, g1.a, K.ey), kh_face_p<float>(w0.a, g0.a, K.ey), kh_face_m<float>(w1.b, g1.b, K.ey),
                      kh_face_p<float>(w0.b, g0.b, K.ey), kh_face_m<float>(w1.d, g1.d, K.ey), kh_face_p<float>(w0.d, g0.d, K.ey),
                      kh_face_m<float>(w1.c, g1.c, K.ey), kh_face_p<float>(w0.c, g0.c, K.ey), r.a, r.b, r.d, r.c);
    return r;
}
__device__ __forceinline__ Row4 kh_row_prim(const Row4& u, const KHK<float>& K)
{
    Row4 w;
    kh_prim_of<float>(u.a, u.b, u.c, u.d, K, w.a, w.b, w.c, w.d);
    return w;
}
// half-step state of a cell
__device__ __forceinline__ Row4 kh_row_prime(const Row4& w, const Row4& gx, const Row4& gy, const KHK<float>& K)
{
    const float gr[8] = {gx.a, gy.a, gx.b, gy.b, gx.c, gy.c, gx.d, gy.d};
    Row4 p;
    kh_prime_of<float>(w.a, w.b, w.c, w.d, gr, K, p.a, p.b, p.c, p.d);
    return p;
}

// a step's constants: those of its dt where the device chooses it (gmax: the maximum after the step
// before it)
__device__ __forceinline__ KHK<float> kh_strip_consts(const KHTileP<float>& P, const unsigned* gmax, double& dt)
{
    KHK<float> K = P.Kc;
    dt = P.dt;
    if (P.cfl > 0.0) {
        dt = P.cfl * P.hmin / (double)__uint_as_float(*gmax);
        K.hdt = (float)(0.5 * dt);
        K.dtdx = (float)(dt * P.dx);
    }
    return K;
}

// half-step state and gradients of cell (x, y) in the step before, in which its block and the ones
// around it were active: from their other buffers, which that step read and nothing has written since
__device__ __forceinline__ Row4 kh_state_before(const GridP& g, const FlagP& f, const KHTileP<float>& P, const KHK<float>& K, int B,
                                                int x, int y, Row4& gx, Row4& gy)
{
    auto prim = [&](int xx, int yy) {
        const int xw = wrap_p(xx, g.nx), yw = wrap_p(yy, g.ny);
        const int par = f.par_cur[xw / B + g.nbx * (yw / B)] ? 0 : 1;
        const size_t gi = (size_t)xw + (size_t)g.nx * yw;
        return kh_row_prim(Row4{P.U[0][par][gi], P.U[1][par][gi], P.U[2][par][gi], P.U[3][par][gi]}, K);
    };
    gx = kh_row_grad(prim(x + 1, y), prim(x - 1, y), K.hx);
    gy = kh_row_grad(prim(x, y + 1), prim(x, y - 1), K.hy);
    return kh_row_prime(prim(x, y), gx, gy, K);
}

// The blocks around block (bx, by) are all set in the flag array w
__device__ __forceinline__ bool kh_around(const GridP& g, const uint8_t* w, int bx, int by)
{
    const int xm = (bx == 0 ? g.nbx : bx) - 1, xp = bx + 1 == g.nbx ? 0 : bx + 1;
    const int ym = ((by == 0 ? g.nby : by) - 1) * g.nbx, yp = (by + 1 == g.nby ? 0 : by + 1) * g.nbx, yc = by * g.nbx;
    // (eight loads in flight, not one after the other)
    const uint8_t a = w[xm + ym], b = w[bx + ym], c = w[xp + ym], d = w[xm + yc], e = w[xp + yc], h = w[xm + yp], i = w[bx + yp], k = w[xp + yp];
    return (a != 0) & (b != 0) & (c != 0) & (d != 0) & (e != 0) & (h != 0) & (i != 0) & (k != 0);
}

// Ring persistence of `cnt` blocks that fell asleep, by the warps of a CTA of 256, half a ring each: what
// their neighbours can read of them (kh_tile_step)
__device__ __forceinline__ void kh_persist_rings(const GridP& g, const FlagP& f, const KHTileP<float>& P, int B, const int* s_blk, int cnt)
{
    double dt;
    const KHK<float> K = kh_strip_consts(P, P.gmax_clear, dt);   // (the maximum that gave the step before its dt)
    const int lane = threadIdx.x & 31;
    for (int j = threadIdx.x >> 5; j < 2 * cnt; j += 8) {
        if (lane >= 2 * B) continue;
        const int bb = s_blk[j >> 1];
        // lanes 0 .. B - 1 the first, B .. 2B - 1 the second side: left column and bottom row, or right
        // column and top row
        const int side = 2 * (j & 1) + lane / B, k = lane % B;
        const int x = (bb % g.nbx) * B + (side == 0 ? 0 : (side == 2 ? B - 1 : k)),
                  y = (bb / g.nbx) * B + (side == 1 ? 0 : (side == 3 ? B - 1 : k));
        const size_t gi = (size_t)x + (size_t)g.nx * y;
        Row4 gx, gy;
        const Row4 p = kh_state_before(g, f, P, K, B, x, y, gx, gy);
        if (side < 2) {
            P.Wp[0][gi] = p.a; P.Wp[1][gi] = p.b; P.Wp[2][gi] = p.c; P.Wp[3][gi] = p.d;
            if (side == 0) {
                P.Gd[0][gi] = gx.a; P.Gd[2][gi] = gx.b; P.Gd[4][gi] = gx.c; P.Gd[6][gi] = gx.d;
            } else {
                P.Gd[1][gi] = gy.a; P.Gd[3][gi] = gy.b; P.Gd[5][gi] = gy.c; P.Gd[7][gi] = gy.d;
            }
        } else {
            Row4 gx1, gy1;
            const Row4 q = kh_state_before(g, f, P, K, B, x + (side == 2), y + (side == 3), gx1, gy1);
            if (side == 2) {
                const Row4 r = kh_row_fx(K, p, gx, q, gx1);
                P.Fl[0][gi] = r.a; P.Fl[1][gi] = r.b; P.Fl[2][gi] = r.c; P.Fl[3][gi] = r.d;
            } else {
                const Row4 r = kh_row_fy(K, p, gy, q, gy1);
                P.Fl[4][gi] = r.a; P.Fl[5][gi] = r.b; P.Fl[6][gi] = r.c; P.Fl[7][gi] = r.d;
            }
        }
    }
}

template <int B, bool DBA>
__global__ void __launch_bounds__(256) kh_strip_scan(GridP g, FlagP f, KHTileP<float> P, KHStripP X)
{
    constexpr int T = 16, TB = T / B, NBT = TB * TB;
    const int ntx = g.nx / T, nty = g.ny / T, ntiles = ntx * nty;
    const int it = blockIdx.x * 256 + threadIdx.x;       // the grid covers the blocks; a tile's on adjacent lanes
    const int tile = it / NBT, kq = it % NBT;
    const bool valid = tile < ntiles;
    const int tby = tile / ntx, tbx = tile - tby * ntx;
    const int bx = tbx * TB + kq % TB, by = tby * TB + kq / TB, b = bx + g.nbx * by;
    const bool cfl = P.cfl > 0.0;
    __shared__ int s_blk[256], s_cnt;                    // blocks that fell asleep since the step before
    __shared__ unsigned s_nw;                            // full tiles
    if (DBA) {
        grid_release();                                  // kh_strip_step may start, and wait
        grid_wait();                                     // the step before
        if (threadIdx.x == 0) {
            s_cnt = 0;
            s_nw = 0u;
        }
        __syncthreads();
    }
    int act = 0, pp = 0;
    bool around = true;                                  // the blocks around this one are active
    bool on = true;
    unsigned vm = 0u;
    if (valid) {
        // (every load that a thread may need in flight at once)
        pp = f.par_cur[b];
        act = DBA ? (f.wake_cur[b] ? 1 : 0) : 1;
        if (DBA) {
            const uint8_t was = X.full[tile];
            on = kh_strips_on(g, X.cnt_prev);
            around = kh_around(g, f.wake_cur, bx, by);
            // fell asleep after a step that took its tile by strips
            if (!act && was) s_blk[atomicAdd(&s_cnt, 1)] = b;
        } else {
            f.wake_nxt[b] = 1;
        }
        f.par_nxt[b] = (uint8_t)(pp ^ act);
        f.wake_clr[b] = 0;
    }
    __syncwarp();                                        // the tile's lanes have read its entry
    count_stats(f.stats, act, valid);
    const unsigned ma = __ballot_sync(0xffffffffu, valid && act);
    const unsigned mr = __ballot_sync(0xffffffffu, valid && act && around);
    const unsigned mp = __ballot_sync(0xffffffffu, valid && pp);
    const int g0 = (threadIdx.x & 31) & ~(NBT - 1);
    constexpr unsigned gm = (1u << NBT) - 1u;
    const unsigned abits = (ma >> g0) & gm, pbits = (mp >> g0) & gm;
    const bool whole = ((mr >> g0) & gm) == gm, full = whole && on;
    if (DBA) {
        const unsigned nw = __popc(__ballot_sync(0xffffffffu, valid && kq == 0 && whole));
        if ((threadIdx.x & 31) == 0 && nw) atomicAdd(&s_nw, nw);
    }
    if (it == 0) {
        *X.cnt_next = 0u;
        *X.taken = 0u;
        if (!DBA) *X.cnt_cur = (unsigned)ntiles;
    }
    if (valid) {
        if (kq == 0) X.full[tile] = full;
        if (DBA && full) f.next[b] = 0;                  // (kh_strip_step sets it)
        if (cfl) {
            if (full) P.vmax[b] = 0.f;                   // kh_strip_step takes the maximum into it
            else if (!act) vm = __float_as_uint(P.vmax[b]);
        }
    }
    if (!DBA) return;
    const int X0 = tbx * T, Y0 = tby * T;
    const bool inner = X0 >= 2 && X0 + T + 2 <= g.nx && Y0 >= 2 && Y0 + T + 2 <= g.ny;
    tile_list_append(f, valid && kq == 0 && abits != 0 && !full, tbx | (tby << 15) | ((int)inner << 30),
                     abits | (pbits << 16), (unsigned)ntiles);
    if (cfl) {
        vm = __reduce_max_sync(0xffffffffu, vm);
        if ((threadIdx.x & 31) == 0 && vm) atomicMax(P.gmax_cur, vm);
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_nw) atomicAdd(X.cnt_cur, s_nw);
    if (s_cnt) kh_persist_rings(g, f, P, B, s_blk, s_cnt);
}

// The rings that the next step's scan would persist, ahead of a save: a saved state holds them, since
// another context that loads it may take its steps with other constants.  By the flags of the step
// before: a ring that the tile kernel has persisted is the same computed again.
template <int B>
__global__ void __launch_bounds__(256) kh_strip_flush(GridP g, FlagP f, KHTileP<float> P)
{
    __shared__ int s_blk[256], s_cnt;
    const int b = blockIdx.x * 256 + threadIdx.x;
    if (threadIdx.x == 0) s_cnt = 0;
    __syncthreads();
    if (b < g.nb && !f.wake_cur[b] && f.wake_clr[b] && kh_around(g, f.wake_clr, b % g.nbx, b / g.nbx)) s_blk[atomicAdd(&s_cnt, 1)] = b;
    __syncthreads();
    if (s_cnt) kh_persist_rings(g, f, P, B, s_blk, s_cnt);
}

// ---- the formulas on pairs of columns (k_pair.cuh): lane by lane the operations, their order
// and their rounding are those of k_kh.cuh ----
struct Pair4 {
    f2 a, b, c, d;
};
// splatted constants
struct KHPairK {
    f2 nz, ivol, gm1, mhalf, half, hx, hy, ex, mex, ey, mey, gam, ig1;
    float gams;
};
inline KHPairK make_kh_pair(const KHK<float>& K)
{
    KHPairK q;
    q.nz = f2_splat_host(-0.f);
    q.ivol = f2_splat_host(K.ivol); q.gm1 = f2_splat_host(K.gm1); q.mhalf = f2_splat_host(-0.5f); q.half = f2_splat_host(0.5f);
    q.hx = f2_splat_host(K.hx); q.hy = f2_splat_host(K.hy);
    q.ex = f2_splat_host(K.ex); q.mex = f2_splat_host(-K.ex); q.ey = f2_splat_host(K.ey); q.mey = f2_splat_host(-K.ey);
    q.gam = f2_splat_host(K.gam); q.ig1 = f2_splat_host(K.ig1);
    q.gams = K.gam;
    return q;
}
__device__ __forceinline__ f2 rcp2(f2 v) { return f2_pack(krcp(f2_lo(v)), krcp(f2_hi(v))); }
// the values one column to the right / left of a lane's two
__device__ __forceinline__ f2 right2(f2 v) { return f2_pack(f2_hi(v), __shfl_down_sync(0xffffffffu, f2_lo(v), 1)); }
__device__ __forceinline__ f2 left2(f2 v) { return f2_pack(__shfl_up_sync(0xffffffffu, f2_hi(v), 1), f2_lo(v)); }
__device__ __forceinline__ Pair4 right4(const Pair4& q) { return Pair4{right2(q.a), right2(q.b), right2(q.c), right2(q.d)}; }
__device__ __forceinline__ Pair4 left4(const Pair4& q) { return Pair4{left2(q.a), left2(q.b), left2(q.c), left2(q.d)}; }

// kh_prim_of
__device__ __forceinline__ Pair4 kh_pair_prim(const KHPairK& K, const Pair4& u)
{
    const f2 iu = rcp2(u.a);
    Pair4 w;
    w.a = mul2(u.a, K.ivol, K.nz);
    w.c = mul2(u.b, iu, K.nz);
    w.d = mul2(u.c, iu, K.nz);
    const f2 ke = fma2(w.c, w.c, mul2(w.d, w.d, K.nz));
    w.b = mul2(K.gm1, fma2(mul2(K.mhalf, w.a, K.nz), ke, mul2(u.d, K.ivol, K.nz)), K.nz);
    return w;
}
__device__ __forceinline__ Pair4 kh_pair_grad(const KHPairK& K, const Pair4& p, const Pair4& m, f2 h)
{
    return Pair4{mul2(sub2(p.a, m.a), h, K.nz), mul2(sub2(p.b, m.b), h, K.nz), mul2(sub2(p.c, m.c), h, K.nz), mul2(sub2(p.d, m.d), h, K.nz)};
}
// kh_prime_of; mh = -dt / 2
__device__ __forceinline__ Pair4 kh_pair_prime(const KHPairK& K, f2 mh, const Pair4& w, const Pair4& gx, const Pair4& gy)
{
    const f2 dv = add2(gx.c, gy.d), ir = rcp2(w.a);
    Pair4 p;
    p.a = fma2(mh, fma2(w.c, gx.a, fma2(w.d, gy.a, mul2(w.a, dv, K.nz))), w.a);
    p.c = fma2(mh, fma2(w.c, gx.c, fma2(w.d, gy.c, mul2(ir, gx.b, K.nz))), w.c);
    p.d = fma2(mh, fma2(w.c, gx.d, fma2(w.d, gy.d, mul2(ir, gy.b, K.nz))), w.d);
    p.b = fma2(mh, fma2(mul2(K.gam, w.b, K.nz), dv, fma2(w.c, gx.b, mul2(w.d, gy.b, K.nz))), w.b);
    return p;
}
// kh_metric of one of the two columns
__device__ __forceinline__ float kh_metric8(float a, float b, float c, float d, float e, float f, float g, float h)
{
    const float gr[8] = {a, b, c, d, e, f, g, h};
    return kh_metric<float>(gr);
}
// kh_getflux; L, R: density, pressure, normal and tangential velocity; outputs Mass, Energy, normal, tangential
__device__ __forceinline__ void kh_pair_flux(const KHPairK& K, const Pair4& L, const Pair4& R, f2& fM, f2& fE, f2& fN, f2& fT)
{
    const f2 nz = K.nz;
    const f2 eL = fma2(mul2(K.half, L.a, nz), fma2(L.c, L.c, mul2(L.d, L.d, nz)), mul2(L.b, K.ig1, nz));
    const f2 eR = fma2(mul2(K.half, R.a, nz), fma2(R.c, R.c, mul2(R.d, R.d, nz)), mul2(R.b, K.ig1, nz));
    const f2 nL = mul2(L.a, L.c, nz), nR = mul2(R.a, R.c, nz), tL = mul2(L.a, L.d, nz), tR = mul2(R.a, R.d, nz);
    const f2 rs = mul2(K.half, add2(L.a, R.a), nz), ns = mul2(K.half, add2(nL, nR), nz), ts = mul2(K.half, add2(tL, tR), nz),
             es = mul2(K.half, add2(eL, eR), nz);
    const f2 irs = rcp2(rs);
    const f2 vs = mul2(ns, irs, nz);
    const f2 ps = mul2(K.gm1, fma2(mul2(K.mhalf, irs, nz), fma2(ns, ns, mul2(ts, ts, nz)), es), nz);
    const f2 cL = mul2(mul2(K.gam, L.b, nz), rcp2(L.a), nz), cR = mul2(mul2(K.gam, R.b, nz), rcp2(R.a), nz);
    const f2 C = f2_pack(fmaxf(__fadd_rn(kq(f2_lo(cL)), fabsf(f2_lo(L.c))), __fadd_rn(kq(f2_lo(cR)), fabsf(f2_lo(R.c)))),
                         fmaxf(__fadd_rn(kq(f2_hi(cL)), fabsf(f2_hi(L.c))), __fadd_rn(kq(f2_hi(cR)), fabsf(f2_hi(R.c)))));
    const f2 mC = mul2(K.mhalf, C, nz);
    fM = fma2(mC, sub2(L.a, R.a), ns);
    fN = fma2(mC, sub2(nL, nR), fma2(ns, vs, ps));
    fT = fma2(mC, sub2(tL, tR), mul2(ts, vs, nz));
    fE = fma2(mC, sub2(eL, eR), mul2(add2(es, ps), vs, nz));
}

template <int B, bool DBA>
__global__ void __launch_bounds__(DBA ? KHStrip::NTD : KHStrip::NT, DBA ? 1 : 4) kh_strip_step(GridP g, FlagP f, KHTileP<float> P, KHStripP X, KHPairK K, int H)
{
    constexpr int OUT = KHStrip::OUT, NT = DBA ? KHStrip::NTD : KHStrip::NT;
    if (DBA) {
        grid_wait();                                     // the scan
        grid_release();                                  // kh_tile_step works on other tiles
        if (!kh_strips_on(g, X.cnt_prev)) return;
    }
    const int lane = threadIdx.x & 31;
    const int nsx = (g.nx + OUT - 1) / OUT;
    // (DBA: consecutive units on different SMs)
    int u = DBA ? (int)(blockIdx.x + gridDim.x * (threadIdx.x >> 5)) : (int)(blockIdx.x * (NT / 32) + (threadIdx.x >> 5));
    const bool cfl = P.cfl > 0.0;
    f2 mh, dtdx;
    {
        double dt;
        const KHK<float> Kd = kh_strip_consts(P, P.gmax_prev, dt);
        mh = f2_pack(-Kd.hdt, -Kd.hdt);
        dtdx = f2_pack(Kd.dtdx, Kd.dtdx);
        if (!DBA && cfl && blockIdx.x == 0 && threadIdx.x == 0) {   // (DBA: kh_tile_step)
            *P.gmax_clear = 0u;
            *P.time += dt;
        }
    }
    unsigned vwarp = 0u;
    bool bad = false;
    // Regular steps: a unit per warp.  DBA: the warps that are resident at once (what a step without strips
    // pays for) take one unit each, and further ones from a counter.
    const int warps = gridDim.x * (NT / 32);
    auto next_unit = [&]() -> int {
        int n = 0;
        if (lane == 0) n = warps + (int)atomicAdd(X.taken, 1u);
        return __shfl_sync(0xffffffffu, n, 0);
    };
    const float thr = (float)P.thr;
    const int ntx = g.nx / 16;
    const size_t nx = (size_t)g.nx;
    for (;; u = next_unit()) {
        const int sy = u / nsx, sx = u - sy * nsx;
        const int y0 = sy * H, rows = min(H, g.ny - y0);
        if (y0 >= g.ny) break;
        const int xr = sx * OUT + 2 * lane - 2;              // the lane's first column; past the grid's last one it is no output
        const bool own = lane >= 1 && lane <= 30 && xr < g.nx;
        int x = wrap_p(xr, g.nx);
        while (x >= g.nx) x -= g.nx;                         // (a narrow grid wraps more than once)
        if (DBA) {                                           // a unit without a full tile has nothing to do
            bool any = false;
            for (int y = y0; y < y0 + rows; y += 16) any |= own && X.full[x / 16 + ntx * (y / 16)];
            if (!__any_sync(0xffffffffu, any)) continue;
        }

        int par = 0;                                         // buffer of the block of the row last loaded
        auto load = [&](int y) -> Pair4 {                    // conserved fields of row y (wrapped), the block's current buffer
            const int yw = wrap_p(y, g.ny);
            if (yw % B == 0 || y < y0 - 1) par = f.par_cur[x / B + g.nbx * (yw / B)] ? 1 : 0;
            const size_t gi = (size_t)x + nx * yw;
            Pair4 q;
            q.a = *reinterpret_cast<const f2*>(P.U[0][par] + gi);
            q.b = *reinterpret_cast<const f2*>(P.U[1][par] + gi);
            q.c = *reinterpret_cast<const f2*>(P.U[2][par] + gi);
            q.d = *reinterpret_cast<const f2*>(P.U[3][par] + gi);
            return q;
        };
        Pair4 up = load(y0 - 2);
        Pair4 wm = kh_pair_prim(K, up);
        up = load(y0 - 1);
        Pair4 wc = kh_pair_prim(K, up);
        up = load(y0);                                       // conserved fields of row y + 1
        Pair4 rm = {}, fd = {}, dfx = {};                    // row y - 1: state at its upper face, flux below it, its x flux difference
        bool hit = false;
        unsigned vblk = 0u;
        bool on = false;                                     // the row being updated: the lane's cells are of a full tile,
        int dst = 0;                                         //   and the buffer they go to
#pragma unroll 1
        for (int y = y0 - 1; y <= y0 + rows; ++y) {
            Pair4 un = up;
            if (y < y0 + rows) un = load(y + 2);             // a row ahead of its use
            Pair4 old = up;                                  // conserved fields of row y - 1, again (L1 holds the last rows)
            if (y > y0) {
                const size_t gi = (size_t)x + nx * (y - 1);
                if ((y - 1) % B == 0) dst = f.par_cur[x / B + g.nbx * ((y - 1) / B)] ? 0 : 1;
                old.a = *reinterpret_cast<const f2*>(P.U[0][dst ^ 1] + gi);
                old.b = *reinterpret_cast<const f2*>(P.U[1][dst ^ 1] + gi);
                old.c = *reinterpret_cast<const f2*>(P.U[2][dst ^ 1] + gi);
                old.d = *reinterpret_cast<const f2*>(P.U[3][dst ^ 1] + gi);
            }
            const Pair4 wp = kh_pair_prim(K, up);
            const Pair4 gx = kh_pair_grad(K, right4(wc), left4(wc), K.hx), gy = kh_pair_grad(K, wp, wm, K.hy);
            const Pair4 pc = kh_pair_prime(K, mh, wc, gx, gy);
            if (y >= y0) {
                Pair4 fu;                                    // the face below row y
                {
                    const Pair4 L{fma2(gy.a, K.mey, pc.a), fma2(gy.b, K.mey, pc.b), fma2(gy.d, K.mey, pc.d), fma2(gy.c, K.mey, pc.c)};
                    kh_pair_flux(K, L, rm, fu.a, fu.b, fu.d, fu.c);
                }
                if (y > y0) {
                    // update of row y - 1
                    const int yr = y - 1;
                    const int b = x / B + g.nbx * (yr / B);
                    if (yr % B == 0) on = own && (!DBA || X.full[x / 16 + ntx * (yr / 16)]);
                    if (on) {
                        const size_t gi = (size_t)x + nx * yr;
                        auto upd = [&](int q, f2 o, f2 d, f2 a, f2 c) -> f2 {   // field q: old value, x flux difference, fluxes above and below
                            const f2 n = add2(o, mul2(dtdx, add2(sub2(d, a), c), K.nz));
                            *reinterpret_cast<f2*>(P.U[q][dst] + gi) = n;
                            return n;
                        };
                        const Pair4 n{upd(0, old.a, dfx.a, fu.a, fd.a), upd(1, old.b, dfx.c, fu.c, fd.c),
                                      upd(2, old.c, dfx.d, fu.d, fd.d), upd(3, old.d, dfx.b, fu.b, fd.b)};
                        // NaN once any stored value is not finite (times a zero from the parameters)
                        const f2 chk = fma2(n.a, K.nz, fma2(n.b, K.nz, fma2(n.c, K.nz, mul2(n.d, K.nz, K.nz))));
                        bad |= !(f2_lo(chk) == 0.f && f2_hi(chk) == 0.f);
                        if (cfl) {
                            const Pair4 w = kh_pair_prim(K, n);
                            vblk = max(vblk, max(__float_as_uint(kh_speed<float>(f2_lo(w.a), f2_lo(w.b), f2_lo(w.c), f2_lo(w.d), K.gams)),
                                                 __float_as_uint(kh_speed<float>(f2_hi(w.a), f2_hi(w.b), f2_hi(w.c), f2_hi(w.d), K.gams))));
                        }
                    }
                    if ((yr + 1) % B == 0) {                 // a block row ends: its blocks' speeds and tests
                        if (cfl) {
                            const unsigned grp = __match_any_sync(0xffffffffu, on ? b : -1);
                            const unsigned v = __reduce_max_sync(grp, vblk);
                            if (on && lane == __ffs(grp) - 1 && v) atomicMax(reinterpret_cast<unsigned*>(P.vmax) + b, v);
                            vwarp = max(vwarp, vblk);
                            vblk = 0u;
                        }
                        if (DBA) {                           // next flag, wake-up of the block and the 8 around it
                            if (on && hit) {
                                const int bx = x / B, by = yr / B;
                                const int xm = (bx == 0 ? g.nbx : bx) - 1, xp = bx + 1 == g.nbx ? 0 : bx + 1;
                                const int ym = ((by == 0 ? g.nby : by) - 1) * g.nbx, yp = (by + 1 == g.nby ? 0 : by + 1) * g.nbx, yc = by * g.nbx;
                                uint8_t* w = f.wake_nxt;
                                f.next[b] = 1;
                                w[xm + ym] = w[bx + ym] = w[xp + ym] = w[xm + yc] = w[b] = w[xp + yc] = w[xm + yp] = w[bx + yp] = w[xp + yp] = 1;
                            }
                            hit = false;
                        }
                    }
                }
                fd = fu;
                if (DBA)                                     // (row y, recorded when its block row is updated)
                    hit |= kh_metric8(f2_lo(gx.a), f2_lo(gy.a), f2_lo(gx.b), f2_lo(gy.b), f2_lo(gx.c), f2_lo(gy.c), f2_lo(gx.d), f2_lo(gy.d)) > thr ||
                           kh_metric8(f2_hi(gx.a), f2_hi(gy.a), f2_hi(gx.b), f2_hi(gy.b), f2_hi(gx.c), f2_hi(gy.c), f2_hi(gx.d), f2_hi(gy.d)) > thr;
                Pair4 fr;
                {
                    const Pair4 m{fma2(gx.a, K.mex, pc.a), fma2(gx.b, K.mex, pc.b), fma2(gx.c, K.mex, pc.c), fma2(gx.d, K.mex, pc.d)};
                    const Pair4 R{fma2(gx.a, K.ex, pc.a), fma2(gx.b, K.ex, pc.b), fma2(gx.c, K.ex, pc.c), fma2(gx.d, K.ex, pc.d)};
                    kh_pair_flux(K, right4(m), R, fr.a, fr.b, fr.c, fr.d);
                }
                const Pair4 fl = left4(fr);
                dfx = Pair4{sub2(fl.a, fr.a), sub2(fl.b, fr.b), sub2(fl.c, fr.c), sub2(fl.d, fr.d)};
            }
            wm = wc; wc = wp;
            up = un;
            rm = Pair4{fma2(gy.a, K.ey, pc.a), fma2(gy.b, K.ey, pc.b), fma2(gy.d, K.ey, pc.d), fma2(gy.c, K.ey, pc.c)};   // (normal velocity third)
        }
        if (!DBA) break;
    }
    if (bad) raise_status(f.status, 5);
    if (cfl) {
        vwarp = __reduce_max_sync(0xffffffffu, vwarp);
        if (lane == 0 && vwarp) atomicMax(P.gmax_cur, vwarp);
    }
}

}  // namespace dba

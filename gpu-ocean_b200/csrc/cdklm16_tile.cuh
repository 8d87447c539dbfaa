// One Runge-Kutta sub-step of CDKLM16 on two-dimensional tiles, with packed
// FP32x2 arithmetic: the stage kernel of small and middle-sized grids.
//
// Restates cdklm_swe_2D (gpu_ocean/SWESimulators/gpu_kernels/CDKLM16_kernel.cu:429-1006)
// followed by the periodic ghost refresh the host issues after it
// (Common.py:1219-1239 -> boundary_kernels.cu:35-110), with the same
// per-operation rounding as the marching and column-pair kernels (their
// helpers are used, so every value is the same bit for bit).
//
// Work layout.  A block of 256 threads writes a tile of 32 x 16 cells.
// Thread (lane, warp w) owns the two cells (column lane, rows w and w + 8) as
// the lanes of float2 values: the rows of a pair lie half a tile apart, so
// the neighbours of a pair in y are the pairs of the next thread rows and
// need no register shuffling, and those in x are the pairs of the next lanes.
// The stage runs in four phases over shared memory (cell states, slopes,
// face fluxes, update); each cell state, slope and face flux of the tile is
// evaluated once, those of the rim by warps 0 .. 7 as a second item.  All
// rows of the tile are in flight together: a marching strip is a serial chain
// of about 1 us per row and primes four rows, which is what a grid of fewer
// cells than the chip has lanes waits for.
//
// Deep tiles.  A tile whose corners and cell states are those of deep water
// (deep.cuh) runs the phases without the scheme's dry, shallow, land and
// zero-fan branches.  The test is one __syncthreads_and in a barrier's place.
// (One form with these branches behind a warp-uniform flag, and the choice of
// the form per warp, both measured slower: 1024^2 49 us per RK2 step, 62 and 55.)
//
// Bounds.  Small grids wait for one tile's chain (loads, four phases) and the
// launch; from about 600^2 cells the kernel is bound by instruction issue and
// by the barriers of the phases: 469 / 486 instructions per cell in stage 0 / 1 (ncu,
// 1024^2), with which the live rate fills 58% of the issue slots; of the warps
// that wait, most wait at barriers.  Scheme factors are kernel arguments
// as pairs, which a packed product takes as one operand (1002 -> 923
// instructions per pair), and all tile arrays share one pitch, so that one
// offset per thread addresses them (1192 -> 1002 with the interior tiles
// compiled without the rim's range tests and signs).
#pragma once

#include <cooperative_groups.h>

#include "cdklm16_pair.cuh"

namespace go {

constexpr int kTileX = 32;                 // columns of a tile, one per lane
constexpr int kTileS = 8;                  // rows between the two cells of a pair (= warps)
constexpr int kTileY = 2 * kTileS;         // rows of a tile
constexpr int kTileThreads = kTileX * kTileS;
// Blocks per SM the kernels are compiled for.  Four (64 registers) measured
// against three (80) for one stage per launch, us per RK2 step on a B200:
// 512^2 17.2 / 19.0 (512 tiles, one wave of four), 768^2 30.7 / 31.2, 1024^2
// 49.2 / 49.8, 1536^2 100 / 103; 640^2 24.3 / 23.5.  The launch of many steps
// runs one tile per SM and needs no spills.
constexpr int kTileBlocks = 4;
constexpr int kTileStepsBlocks = 2;

// Launch constants of the tile kernels: the scheme's factors as pairs, which packed products take as one operand.
struct TileConst {
    float2 theta, half, theta_g, half_g, mV, U, g, two;
};
inline TileConst tile_const(const Scheme& k) {
    auto b = [](float s) { return make_float2(s, s); };
    return TileConst{b(k.theta), b(0.5f), b(k.theta_g), b(k.half_g), b(-k.V), b(k.U), b(k.g), b(2.0f)};
}
// Shared memory of one tile.  State row p holds the row pair (k, k + 8) with
// k = p - 2, column q the tile column q - 2; every array has the same pitch,
// so that one offset at(p, q) per thread serves them all, and is trimmed to the
// rows its phase needs (first row in the name's comment).
constexpr int kTilePitch = kTileX + 6;
__device__ __forceinline__ constexpr int tile_at(int p, int q) { return p * kTilePitch + q; }

struct TileSmem {
    float4 eu[(kTileS + 4) * kTilePitch];     // (eta, eta, u, u); p = 0
    float4 xs_[kTileS * kTilePitch];          // x slopes (u, u, v, v); p = 2
    float4 ys_[(kTileS + 2) * kTilePitch];    // y slopes (u, u, v, v); p = 1
    float4 F01_[kTileS * kTilePitch];         // (F0, F0, F1, F1) on the west faces; p = 2
    float4 G01_[(kTileS + 1) * kTilePitch];   // (G0, G0, G1, G1) on the south faces; p = 2
    float2 H[(kTileS + 5) * kTilePitch];      // corners south-west of the cells; p = 0
    float2 v[(kTileS + 4) * kTilePitch];
    float2 fu[(kTileS + 4) * kTilePitch];     // f u' of the y slopes, f v' of the x slopes
    float2 fv[(kTileS + 4) * kTilePitch];     // (u', v' turned in wall ghost cells)
    float2 xk_[kTileS * kTilePitch];          // K; p = 2
    float2 yl_[(kTileS + 2) * kTilePitch];    // L; p = 1
    float2 F2_[kTileS * kTilePitch];          // p = 2
    float2 G2_[(kTileS + 1) * kTilePitch];    // p = 2
    float2 f[kTileS + 4];                     // Coriolis parameter of the row pairs
    // element of a trimmed array at offset o = tile_at(p, q)
    __device__ __forceinline__ float4& xs(int o) { return xs_[o - 2 * kTilePitch]; }
    __device__ __forceinline__ float4& ys(int o) { return ys_[o - kTilePitch]; }
    __device__ __forceinline__ float4& F01(int o) { return F01_[o - 2 * kTilePitch]; }
    __device__ __forceinline__ float4& G01(int o) { return G01_[o - 2 * kTilePitch]; }
    __device__ __forceinline__ float2& xk(int o) { return xk_[o - 2 * kTilePitch]; }
    __device__ __forceinline__ float2& yl(int o) { return yl_[o - kTilePitch]; }
    __device__ __forceinline__ float2& F2(int o) { return F2_[o - 2 * kTilePitch]; }
    __device__ __forceinline__ float2& G2(int o) { return G2_[o - 2 * kTilePitch]; }
};

// A value that is the same in all lanes of the warp, so that the compiler knows
// it too: branches on it then need no reconvergence point and leave uniform
// registers in use (warp index and votes through this: 252 -> 172 bytes of
// spills, us per RK2 step 512^2 17.3 -> 16.6, 1024^2 48.8 -> 48.0).
__device__ __forceinline__ int warp_uniform(int x) { return __shfl_sync(0xffffffffu, x, 0); }

__device__ __forceinline__ float2 lo2(float4 a) { return make_float2(a.x, a.y); }
__device__ __forceinline__ float2 hi2(float4 a) { return make_float2(a.z, a.w); }
__device__ __forceinline__ float4 cat4(float2 a, float2 b) { return make_float4(a.x, a.y, b.x, b.y); }
// lane-wise product, two scalar multiplies (see pscale)
__device__ __forceinline__ float2 plane(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }

// minmodSlope (common.cu:532-542) per lane, packed products.
__device__ __forceinline__ float2 tile_slope(float2 l, float2 c, float2 r, const TileConst& tc, float2 nz) {
    return pminmod(pmul_nz(psub(c, l), tc.theta, nz), pmul_nz(psub(r, l), tc.half, nz),
                   pmul_nz(psub(r, c), tc.theta, nz));
}

// The tile of one block: its first written cell, and the source cell and
// sign of a ghost-inclusive row or column (walls mirror the interior with
// the normal momentum turned; cells past the array clamp, feed no written
// cell and are never written).
struct TilePlace {
    int c0, r0;          // ghost-inclusive column and row of the tile's first cell
    bool rim;            // the tile or its halo reaches ghost cells or the array's end
};

__device__ __forceinline__ TilePlace tile_place(const Scheme& k, int bx, int by) {
    TilePlace t;
    t.c0 = 2 + bx * kTileX;
    t.r0 = 2 + by * kTileY;
    t.rim = bx == 0 || by == 0 || t.c0 + kTileX + 2 > k.nx + 2 || t.r0 + kTileY + 2 > k.ny + 2;
    return t;
}

__device__ __forceinline__ int tile_src(int i, int n, bool wall_lo, bool wall_hi, float& sign) {
    sign = 1.0f;
    if (wall_lo && i < 2) { sign = -1.0f; return 3 - i; }
    if (wall_hi && i > n + 1 && i <= n + 3) { sign = -1.0f; return 2 * n + 3 - i; }
    return min(i, n + 3);
}

// Address a byte offset beyond a base: a 32-bit offset adds to a uniform base
// in the load or store itself.  (A tile launch's arrays are below 4 GB.)
__device__ __forceinline__ const float* at_byte(const float* p, unsigned b) {
    return reinterpret_cast<const float*>(reinterpret_cast<const char*>(p) + b);
}
__device__ __forceinline__ float* at_byte(float* p, unsigned b) {
    return reinterpret_cast<float*>(reinterpret_cast<char*>(p) + b);
}

// Corners and Coriolis rows of a tile into shared memory; returns whether
// this thread's values allow a deep tile.  No barrier.
template <bool RIM>
__device__ __forceinline__ bool tile_load_fixed(const StageArgs& a, const TilePlace& t, TileSmem& sm) {
    const Scheme& k = a.k;
    const int lane = threadIdx.x & 31, w = warp_uniform((int)threadIdx.x >> 5);
    const long long xhi = ext_hi(a), xf = ext_f(a);
    const float hi = deep_end(k);
    bool ok = true;
    auto corner_at = [&](int r, int c) {
        const int rr = RIM ? min(t.r0 - 2 + r, k.ny + 4) : t.r0 - 2 + r;
        const int cc = RIM ? min(t.c0 - 2 + c, k.nx + 4) : t.c0 - 2 + c;
        const unsigned o = (unsigned)rr * (unsigned)a.phi + (unsigned)cc;
        return idx_ok(o, 1, xhi, a.status) ? __ldg(at_byte(a.Hi, 4u * o)) : 0.0f;
    };
    auto keep = [&](int r, int c, float h) {
        ok = ok && h >= a.deep_lo && h < hi;
        const float hc = corner(h, k);
        if (r < kTileS + 5) sm.H[tile_at(r, c)].x = hc;
        if (r >= kTileS) sm.H[tile_at(r - kTileS, c)].y = hc;
    };
    // rows w, w + 8 and (w < 5) w + 16, 37 columns: the lanes' column and 5 more
    const float h0 = corner_at(w, lane), h1 = corner_at(w + kTileS, lane);
    const float h2 = w < 5 ? corner_at(w + 2 * kTileS, lane) : 0.0f;
    const int r3 = threadIdx.x / 5, c3 = kTileX + threadIdx.x % 5;
    const float h3 = r3 < kTileY + 5 ? corner_at(r3, c3) : 0.0f;
    keep(w, lane, h0);
    keep(w + kTileS, lane, h1);
    if (w < 5) keep(w + 2 * kTileS, lane, h2);
    if (r3 < kTileY + 5) keep(r3, c3, h3);
    if (threadIdx.x < kTileS + 4) {
        const int r = t.r0 - 2 + (int)threadIdx.x;
        const float2 f = make_float2(ldg1(a.f_rows, min(r, k.ny + 3), xf, a.status),
                                     ldg1(a.f_rows, min(r + kTileS, k.ny + 3), xf, a.status));
        sm.f[threadIdx.x] = f;
        ok = ok && fabsf(f.x) <= a.deep_f && fabsf(f.y) <= a.deep_f;
    }
    return ok;
}

// Inputs of the cell pair at state row p, column q.
struct TileQ {
    float2 e, hu, hv;
};

// The states a stage reads and writes, and the state before the step that
// stage 1 reads at the cells it writes.
struct TileIO {
    const float *e, *hu, *hv;
    float *oe, *ohu, *ohv;
    const float *ne, *nhu, *nhv;
    int pin, pout, pn;       // pitches, floats
};

template <bool RIM>
__device__ __forceinline__ TileQ tile_load_q(const StageArgs& a, const TileIO& io, const TilePlace& t, int p, int q) {
    const Scheme& k = a.k;
    const long long xin = (long long)(k.ny + 4) * io.pin;
    const int c = t.c0 - 2 + q, r = t.r0 - 2 + p;
    TileQ Q;
    auto ld = [&](const float* s, unsigned o) {
        return idx_ok(o, 1, xin, a.status) ? __ldcg(at_byte(s, 4u * o)) : 0.0f;
    };
    if (RIM) {
        float sc, sx, sy;
        const unsigned cc = tile_src(c, k.nx, k.bcW == kWall, k.bcE == kWall, sc);
        const unsigned ox = (unsigned)tile_src(r, k.ny, k.bcS == kWall, k.bcN == kWall, sx) * (unsigned)io.pin + cc;
        const unsigned oy =
            (unsigned)tile_src(r + kTileS, k.ny, k.bcS == kWall, k.bcN == kWall, sy) * (unsigned)io.pin + cc;
        Q.e = make_float2(ld(io.e, ox), ld(io.e, oy));
        Q.hu = make_float2(ld(io.hu, ox) * sc, ld(io.hu, oy) * sc);
        Q.hv = make_float2(ld(io.hv, ox) * sx, ld(io.hv, oy) * sy);
    } else {
        const unsigned ox = (unsigned)r * (unsigned)io.pin + (unsigned)c, oy = ox + kTileS * (unsigned)io.pin;
        Q.e = make_float2(ld(io.e, ox), ld(io.e, oy));
        Q.hu = make_float2(ld(io.hu, ox), ld(io.hu, oy));
        Q.hv = make_float2(ld(io.hv, ox), ld(io.hv, oy));
    }
    return Q;
}

// Reconstruction state of the pair at (p, q) into shared memory and the
// return value; `deep` tells that no corner of the tile is shallow or land.
// Returns whether the pair allows a deep tile.
template <bool RIM>
__device__ __forceinline__ bool tile_cell(const StageArgs& a, const TilePlace& t, TileSmem& sm, int p, int q,
                                          const TileQ& Q, bool deep, float2 NZ, float2& e, float2& u, float2& v) {
    const Scheme& k = a.k;
    const int o = tile_at(p, q);
    const float2 h00 = sm.H[o], h10 = sm.H[o + kTilePitch], h01 = sm.H[o + 1], h11 = sm.H[o + kTilePitch + 1];
    const float2 s = padd(padd(padd(h00, h10), h01), h11);
    float2 Bm = pscale(s, 0.25f);
    if (!deep)
        Bm = make_float2(cell_bm(h00.x, h10.x, h01.x, h11.x, s.x, k), cell_bm(h00.y, h10.y, h01.y, h11.y, s.y, k));
    const float2 h = padd(Q.e, Bm);
    bool wet = h.x >= k.desing_eps && h.y >= k.desing_eps;
    if (!deep) wet = wet && !(fabsf(Bm.x - k.land) <= kDryEps) && !(fabsf(Bm.y - k.land) <= kDryEps);
    if (wet) {
        const float2 rh = make_float2(rcp_approx(h.x), rcp_approx(h.y));
        e = Q.e;
        u = pmul_nz(Q.hu, rh, NZ);
        v = pmul_nz(Q.hv, rh, NZ);
    } else {
        cell_lane<true, true>(Q.e.x, Q.hu.x, Q.hv.x, Bm.x, k, e.x, u.x, v.x);
        cell_lane<true, true>(Q.e.y, Q.hu.y, Q.hv.y, Bm.y, k, e.y, u.y, v.y);
    }
    const float2 f = sm.f[p];
    // u' and v' of the Coriolis terms are turned in wall ghost cells (:633-641, :738-748)
    float2 fu = f, fv = f;
    if (RIM) {
        const int c = t.c0 - 2 + q, r = t.r0 - 2 + p;
        if ((k.bcW == kWall && c < 2) || (k.bcE == kWall && c > k.nx + 1)) fv = make_float2(-fv.x, -fv.y);
        auto turned = [&](int rr) { return (k.bcS == kWall && rr < 2) || (k.bcN == kWall && rr > k.ny + 1); };
        if (turned(r)) fu.x = -fu.x;
        if (turned(r + kTileS)) fu.y = -fu.y;
    }
    sm.eu[o] = cat4(e, u);
    sm.v[o] = v;
    sm.fu[o] = plane(u, fu);
    sm.fv[o] = plane(v, fv);
    return deep_state(e.x, u.x, v.x, a.deep_eta) && deep_state(e.y, u.y, v.y, a.deep_eta);
}

// Slopes of the pair at offset o along one axis: of its velocities and of the
// Coriolis potential (K in x, L in y).  The neighbours' states come from
// shared memory, d the step to the next cell of the axis; sV is -V in
// x (K subtracts V (f v)) and U in y; f* are the Coriolis products of the axis.
// turn: -dx f v' (x) or dy f u' (y) of the slope adjustment (:148-241), which
// is K + dx f v' = K - turn, L - dy f u' = L - turn, with fallbacks
// turn + 2g (..) and turn - 2g (..); Hlo, Hhi the face depths either side.
template <bool DEEP>
__device__ __forceinline__ void tile_slopes(const TileSmem& sm, const float2* fq, int o, int d, float2 e, float2 u,
                                            float2 v, float2 fc, float2 sV, float2 turn, float2 Hlo, float2 Hhi,
                                            const Scheme& k, const TileConst& tc, float2 by2g, float2 NZ, float2& du,
                                            float2& dv, float2& K) {
    const float4 l = sm.eu[o - d], r = sm.eu[o + d];
    const float2 le = lo2(l), re = lo2(r);
    auto pmul = [&](float2 x, float2 y) { return pmul_nz(x, y, NZ); };
    du = tile_slope(hi2(l), u, hi2(r), tc, NZ);
    dv = tile_slope(sm.v[o - d], v, sm.v[o + d], tc, NZ);
    const float2 lf = fq[o - d], rf = fq[o + d];
    const float2 backward = pmul(padd(psub(e, le), pmul(padd(fc, lf), sV)), tc.theta_g);
    const float2 central = pmul(padd(psub(re, le), pmul(padd(padd(rf, pmul(fc, tc.two)), lf), sV)), tc.half_g);
    const float2 forward = pmul(padd(psub(re, e), pmul(padd(fc, rf), sV)), tc.theta_g);
    K = pminmod(backward, central, forward);
    if (!DEEP) {
        const float2 dq2 = pmul(psub(K, turn), by2g);
        const float2 lo = psub(padd(e, Hlo), dq2), hi = padd(padd(e, Hhi), dq2);
        auto fix = [&](float Kv, float tv, float ce, float Hl, float Hh, float lov, float hiv) {
            Kv = (lov > 0.0f) ? Kv : tv + k.two_g * (ce + Hl);
            Kv = (hiv > 0.0f) ? Kv : tv - k.two_g * (ce + Hh);
            return Kv;
        };
        K = make_float2(fix(K.x, turn.x, e.x, Hlo.x, Hhi.x, lo.x, hi.x),
                        fix(K.y, turn.y, e.y, Hlo.y, Hhi.y, lo.y, hi.y));
    }
}

// Flux through the face between the pairs m (low side) and p (high side) of
// an axis: eta, normal and tangential velocity a, b, their slopes and the
// potential's; cm, cp: the Coriolis part of the face depths, added to K
// (dx f v in x, -dy f u in y); H the face depth.
template <bool DEEP>
__device__ __forceinline__ void tile_face(float2 em, float2 am, float2 bm, float2 dam, float2 dbm, float2 Km,
                                          float2 cm, float2 ep, float2 ap, float2 bp, float2 dap, float2 dbp,
                                          float2 Kp, float2 cp, float2 H, const Scheme& k, const TileConst& tc,
                                          float2 by2g, float2 NZ, float2& F0, float2& F1, float2& F2) {
    auto pmul = [&](float2 x, float2 y) { return pmul_nz(x, y, NZ); };
    const float2 hp = psub(padd(ep, H), pmul(padd(Kp, cp), by2g));
    const float2 hm = padd(padd(em, H), pmul(padd(Km, cm), by2g));
    const float2 ua = padd(am, pmul(dam, tc.half)), ub = padd(bm, pmul(dbm, tc.half));
    const float2 pa = psub(ap, pmul(dap, tc.half)), pb_ = psub(bp, pmul(dbp, tc.half));
    if (DEEP) {
        pflux_deep(hm, ua, ub, hp, pa, pb_, tc.half_g, tc.g, NZ, F0, F1, F2);
    } else {
        pflux<true>(make_float2(fmaxf(0.0f, hm.x), fmaxf(0.0f, hm.y)), ua, ub,
                    make_float2(fmaxf(0.0f, hp.x), fmaxf(0.0f, hp.y)), pa, pb_, k, NZ, F0, F1, F2);
        const bool x = em.x == kDryFlag || ep.x == kDryFlag, y = em.y == kDryFlag || ep.y == kDryFlag;
        const float2 z = pb(0.0f);   // a land cell on either side: zero flux (:271-273)
        F0 = psel(x, y, z, F0); F1 = psel(x, y, z, F1); F2 = psel(x, y, z, F2);
    }
}

// Phases 2 to 4 of a tile whose states lie in shared memory: slopes, fluxes,
// update and store.
template <bool DEEP, bool RIM>
__device__ __forceinline__ void tile_phases(const StageArgs& a, const TileConst& tc, const TileIO& io, const float dt,
                                            const bool stage1, const TilePlace& t, TileSmem& sm, const float2 e,
                                            const float2 u, const float2 v) {
    const Scheme& k = a.k;
    const int lane = threadIdx.x & 31, w = warp_uniform((int)threadIdx.x >> 5);
    const float2 NZ = pb(a.neg_zero);
    auto pmul = [&](float2 x, float2 y) { return pmul_nz(x, y, NZ); };
    const PDiv<true> bydx(k.dx, NZ), bydy(k.dy, NZ);
    const float2 by2g = pb(rcp_approx(k.two_g));
    const bool wW = RIM && k.bcW == kWall, wE = RIM && k.bcE == kWall;
    const bool wS = RIM && k.bcS == kWall, wN = RIM && k.bcN == kWall;
    // dx f and dy f of a row pair, with the signs of the wall ghost cells
    auto dxf = [&](int p) { const float2 f = sm.f[p]; return make_float2(k.dx * f.x, k.dx * f.y); };
    auto dyf = [&](int p) { const float2 f = sm.f[p]; return make_float2(k.dy * f.x, k.dy * f.y); };
    auto flip2 = [](bool x, bool y, float2 s) { return make_float2(x ? -s.x : s.x, y ? -s.y : s.y); };
    // face depths west and south of the cell pair at offset o
    auto Hwest = [&](int o) { return pmul(padd(sm.H[o], sm.H[o + kTilePitch]), tc.half); };
    auto Hsouth = [&](int o) { return pmul(padd(sm.H[o], sm.H[o + 1]), tc.half); };

    auto xslopes = [&](int p, int q, float2 ce, float2 cu, float2 cv, float2& du, float2& dv, float2& K) {
        const int o = tile_at(p, q), c = t.c0 - 2 + q;
        const bool turned = (wW && c < 2) || (wE && c > k.nx + 2);   // :172-174
        float2 turn = pb(0.0f), Hlo = turn, Hhi = turn;
        if (!DEEP) {
            turn = plane(cv, flip2(!turned, !turned, dxf(p)));
            Hlo = Hwest(o);
            Hhi = Hwest(o + 1);
        }
        tile_slopes<DEEP>(sm, sm.fv, o, 1, ce, cu, cv, sm.fv[o], tc.mV, turn, Hlo, Hhi, k, tc, by2g, NZ, du, dv, K);
        sm.xs(o) = cat4(du, dv);
        sm.xk(o) = K;
    };
    auto yslopes = [&](int p, int q, float2 ce, float2 cu, float2 cv, float2& du, float2& dv, float2& L) {
        const int o = tile_at(p, q), r = t.r0 - 2 + p;
        auto turned = [&](int rr) { return (wS && rr < 2) || (wN && rr > k.ny + 2); };
        float2 turn = pb(0.0f), Hlo = turn, Hhi = turn;
        if (!DEEP) {
            turn = plane(cu, flip2(turned(r), turned(r + kTileS), dyf(p)));
            Hlo = Hsouth(o);
            Hhi = Hsouth(o + kTilePitch);
        }
        tile_slopes<DEEP>(sm, sm.fu, o, kTilePitch, ce, cu, cv, sm.fu[o], tc.U, turn, Hlo, Hhi, k, tc, by2g, NZ, du,
                          dv, L);
        sm.ys(o) = cat4(du, dv);
        sm.yl(o) = L;
    };
    // ---- slopes ------------------------------------------------------------
    const int p = w + 2, q = lane + 2, own = tile_at(p, q);
    float2 xu, xv, K, yu, yv, L;
    xslopes(p, q, e, u, v, xu, xv, K);
    yslopes(p, q, e, u, v, yu, yv, L);
    if (w == 5 || w == 6) {              // the rows beside the tile
        const int pr = (w == 5) ? 1 : kTileS + 2, o = tile_at(pr, q);
        const float4 c = sm.eu[o];
        float2 d0, d1, d2;
        yslopes(pr, q, lo2(c), hi2(c), sm.v[o], d0, d1, d2);
    } else if (w == 7 && lane < 2 * kTileS) {   // the columns beside the tile
        const int pr = 2 + (lane >> 1), qc = (lane & 1) ? kTileX + 2 : 1, o = tile_at(pr, qc);
        const float4 c = sm.eu[o];
        float2 d0, d1, d2;
        xslopes(pr, qc, lo2(c), hi2(c), sm.v[o], d0, d1, d2);
    }
    __syncthreads();

    // ---- fluxes through the west and south faces -------------------------------
    auto xface = [&](int pr, int qc, float2 pe, float2 pu, float2 pv, float2 pdu, float2 pdv, float2 pK, float2& F0,
                     float2& F1, float2& F2) {
        const int o = tile_at(pr, qc), c = t.c0 - 2 + qc;
        const float4 m = sm.eu[o - 1], ms = sm.xs(o - 1);
        const float2 mv = sm.v[o - 1], s = dxf(pr);
        const bool fm = wW && c == 2, fp = wE && c == k.nx + 2;      // :286, :288
        tile_face<DEEP>(lo2(m), hi2(m), mv, lo2(ms), hi2(ms), sm.xk(o - 1), plane(mv, flip2(fm, fm, s)), pe, pu, pv,
                        pdu, pdv, pK, plane(pv, flip2(fp, fp, s)), Hwest(o), k, tc, by2g, NZ, F0, F1, F2);
        sm.F01(o) = cat4(F0, F1);
        sm.F2(o) = F2;
    };
    auto yface = [&](int pr, int qc, float2 pe, float2 pu, float2 pv, float2 pdu, float2 pdv, float2 pL, float2& G0,
                     float2& G1, float2& G2) {
        const int o = tile_at(pr, qc), om = o - kTilePitch, r = t.r0 - 2 + pr;
        const float4 m = sm.eu[om], ms = sm.ys(om);
        const float2 mv = sm.v[om], mu = hi2(m);
        const float2 sm_ = dyf(pr - 1), sp = dyf(pr);
        auto fm = [&](int rr) { return !(wS && rr == 2); };          // subtracted: turned twice at a wall
        auto fp = [&](int rr) { return !(wN && rr == k.ny + 2); };
        tile_face<DEEP>(lo2(m), mv, mu, hi2(ms), lo2(ms), sm.yl(om), plane(mu, flip2(fm(r), fm(r + kTileS), sm_)), pe,
                        pv, pu, pdv, pdu, pL, plane(pu, flip2(fp(r), fp(r + kTileS), sp)), Hsouth(o), k, tc, by2g, NZ,
                        G0, G2, G1);
        sm.G01(o) = cat4(G0, G1);
        sm.G2(o) = G2;
    };
    // the state before the step, in flight while the fluxes are computed
    const int col = t.c0 + lane, row = t.r0 + w;
    const bool wr_x = !RIM || (col <= k.nx + 1 && row <= k.ny + 1);
    const bool wr_y = !RIM || (col <= k.nx + 1 && row + kTileS <= k.ny + 1);
    TileQ qn{};
    if (stage1) {
        const long long xn = (long long)(k.ny + 4) * io.pn;
        const unsigned ox = (unsigned)row * (unsigned)io.pn + (unsigned)col, oy = ox + kTileS * (unsigned)io.pn;
        auto ld = [&](const float* s, unsigned o, bool on) {
            return on && idx_ok(o, 1, xn, a.status) ? __ldcg(at_byte(s, 4u * o)) : 0.0f;
        };
        qn.e = make_float2(ld(io.ne, ox, wr_x), ld(io.ne, oy, wr_y));
        qn.hu = make_float2(ld(io.nhu, ox, wr_x), ld(io.nhu, oy, wr_y));
        qn.hv = make_float2(ld(io.nhv, ox, wr_x), ld(io.nhv, oy, wr_y));
    }
    float2 F0, F1, F2, G0, G1, G2;
    xface(p, q, e, u, v, xu, xv, K, F0, F1, F2);
    yface(p, q, e, u, v, yu, yv, L, G0, G1, G2);
    if (w == 0) {                         // the faces north of the tile
        const int o = tile_at(kTileS + 2, q);
        const float4 c = sm.eu[o], s = sm.ys(o);
        float2 d0, d1, d2;
        yface(kTileS + 2, q, lo2(c), hi2(c), sm.v[o], lo2(s), hi2(s), sm.yl(o), d0, d1, d2);
    } else if (w == 1 && lane < kTileS) {   // and east of it
        const int o = tile_at(2 + lane, kTileX + 2);
        const float4 c = sm.eu[o], s = sm.xs(o);
        float2 d0, d1, d2;
        xface(2 + lane, kTileX + 2, lo2(c), hi2(c), sm.v[o], lo2(s), hi2(s), sm.xk(o), d0, d1, d2);
    }
    __syncthreads();

    // ---- update of the own pair (:807-1004) -----------------------------------
    if (!wr_x) return;                    // then neither cell of the pair is written
    const float4 Fe = sm.F01(own + 1), Gn = sm.G01(own + kTilePitch);
    const float2 fd0 = padd(bydx(psub(lo2(Fe), F0)), bydy(psub(lo2(Gn), G0)));
    const float2 fd1 = padd(bydx(psub(hi2(Fe), F1)), bydy(psub(hi2(Gn), G1)));
    const float2 fd2 = padd(bydx(psub(sm.F2(own + 1), F2)), bydy(psub(sm.G2(own + kTilePitch), G2)));
    const float2 h00 = sm.H[own], h10 = sm.H[own + kTilePitch], h01 = sm.H[own + 1], h11 = sm.H[own + kTilePitch + 1];
    const float2 Hm = pscale(padd(padd(padd(h00, h10), h01), h11), 0.25f);
    const float2 f = sm.f[p];
    // face values of eta for the bathymetry source (:706-707, :803-804)
    const float2 ttx = pmul(padd(K, plane(v, dxf(p))), by2g);
    const float2 tty = pmul(psub(L, plane(u, dyf(p))), by2g);
    const float2 h = padd(e, Hm);
    float2 hu = pmul(u, h), hv = pmul(v, h);
    if (!DEEP) {
        hu = psel(h.x > k.cutoff, h.y > k.cutoff, hu, pb(0.0f));
        hv = psel(h.x > k.cutoff, h.y > k.cutoff, hv, pb(0.0f));
    }
    float2 Xv, Yv;
    if (a.wx_cur != nullptr) {
        const long long xw = ext_w(a);
        auto wl = [&](const float* cur, const float* nxt, bool on, int r) {
            if (!on) return 0.0f;
            const size_t o = (size_t)(r - 2) * a.pw + (col - 2);
            const float xn = ldg1(nxt, o, xw, a.status);
            const float xc = (cur == nxt) ? xn : ldg1(cur, o, xw, a.status);
            return a.wind_t * xn + (1.0f - a.wind_t) * xc;
        };
        Xv = make_float2(wl(a.wx_cur, a.wx_next, true, row), wl(a.wx_cur, a.wx_next, wr_y, row + kTileS));
        Yv = make_float2(wl(a.wy_cur, a.wy_next, true, row), wl(a.wy_cur, a.wy_next, wr_y, row + kTileS));
    } else {
        Xv = pb(a.wind_t * a.wxn + (1.0f - a.wind_t) * a.wxc);
        Yv = pb(a.wind_t * a.wyn + (1.0f - a.wind_t) * a.wyc);
    }
    const float2 ew = psub(e, ttx), ee = padd(e, ttx);
    const float2 es = psub(e, tty), en = padd(e, tty);
    const float2 Hx = psub(pmul(padd(h01, h11), tc.half), pmul(padd(h00, h10), tc.half));
    const float2 Hy = psub(pmul(padd(h10, h11), tc.half), pmul(padd(h00, h01), tc.half));
    const float2 bbx = pmul(pmul(padd(pmul(padd(ew, ee), tc.half), Hm), tc.g), Hx);
    const float2 bby = pmul(pmul(padd(pmul(padd(es, en), tc.half), Hm), tc.g), Hy);
    float2 stx = padd(padd(Xv, plane(hv, f)), bydx(bbx));
    float2 sty = padd(padd(Yv, plane(hu, make_float2(-f.x, -f.y))), bydy(bby));
    if (!DEEP) {
        const bool sx = h.x >= k.cutoff && e.x != kDryFlag, sy = h.y >= k.cutoff && e.y != kDryFlag;
        stx = psel(sx, sy, stx, pb(0.0f));
        sty = psel(sx, sy, sty, pb(0.0f));
    }
    const float2 L2 = psub(stx, fd1), L3 = psub(sty, fd2);

    float2 C = pb(0.0f);
    if (a.fric == kFricLinear) {
        C = prcp_or_div<true>(pb(k.two_r * dt), h, NZ);
    } else if (a.fric == kFricQuad) {
        const float dtr = dt * k.r;
        if (DEEP || (h.x >= k.desing_eps && h.y >= k.desing_eps)) {
            const float2 rh = make_float2(rcp_approx(h.x), rcp_approx(h.y));
            const float2 uu = pmul(hu, rh), vv = pmul(hv, rh);
            const float2 ss = padd(pmul(uu, uu), pmul(vv, vv));
            C = pmul(pscale(make_float2(sqrtf(ss.x), sqrtf(ss.y)), dtr), rh);
        } else {
            auto one = [&](float h1, float hu1, float hv1) {
                if (h1 < k.desing_eps) {
                    const float uu = desingularize(h1, hu1, k.desing_eps), vv = desingularize(h1, hv1, k.desing_eps);
                    return dt * k.r * desingularize(h1, sqrtf(uu * uu + vv * vv), k.desing_eps);
                }
                const float uu = quot<true>(hu1, h1), vv = quot<true>(hv1, h1);
                return quot<true>(dtr * sqrtf(uu * uu + vv * vv), h1);
            };
            C = make_float2(one(h.x, hu.x, hv.x), one(h.y, hu.y, hv.y));
        }
    }
    float2 ne = psub(e, pscale(fd0, dt)), bu = padd(hu, pscale(L2, dt)), bv = padd(hv, pscale(L3, dt));
    if (stage1) {
        ne = pmul(padd(qn.e, ne), tc.half);
        bu = pmul(padd(qn.hu, bu), tc.half);
        bv = pmul(padd(qn.hv, bv), tc.half);
        C = pmul(C, tc.half);
    }
    const float2 den = padd(pb(1.0f), C);
    const float2 rden = make_float2(rcp_approx(den.x), rcp_approx(den.y));
    float2 nhu = pmul(bu, rden), nhv = pmul(bv, rden);
    const float2 lim = psub(pb(k.cutoff), Hm);   // -Hm + cutoff
    const float2 hn = padd(ne, Hm);
    const bool dryx = hn.x <= k.cutoff, dryy = hn.y <= k.cutoff;
    if (dryx || dryy) {
        ne = psel(dryx, dryy, lim, ne);
        nhu = psel(dryx, dryy, pb(0.0f), nhu);
        nhv = psel(dryx, dryy, pb(0.0f), nhv);
    }
    ne = make_float2(fmaxf(lim.x, ne.x), fmaxf(lim.y, ne.y));
    const float2 chk = padd(padd(ne, nhu), nhv);
    if (a.status && (!isfinite(chk.x) || (wr_y && !isfinite(chk.y)))) atomicOr(a.status, 1u);

    const long long xout = (long long)(k.ny + 4) * io.pout;
    auto put = [&](int r, int c, float e1, float u1, float v1) {
        const unsigned o = (unsigned)r * (unsigned)io.pout + (unsigned)c;
        if (!idx_ok(o, 1, xout, a.status)) return;
        *at_byte(io.oe, 4u * o) = e1;
        *at_byte(io.ohu, 4u * o) = u1;
        *at_byte(io.ohv, 4u * o) = v1;
    };
    put(row, col, ne.x, nhu.x, nhv.x);
    if (wr_y) put(row + kTileS, col, ne.y, nhu.y, nhv.y);
    if (RIM && (k.bcN == kPeriodic || k.bcE == kPeriodic)) {
        // periodic ghost images (the reference's BC kernels after the stage)
        auto image = [&](int i, int n, bool periodic) {
            if (!periodic) return -1;
            return i < 4 ? i + n : (i >= n ? i - n : -1);
        };
        auto images = [&](int r, float e1, float u1, float v1) {
            // a side shorter than its ghost frame has two images per cell
            for (int ri = -1; ri < 2; ++ri) {
                int rr = r;
                if (ri == 0) rr = image(r, k.ny, k.bcN == kPeriodic);
                if (ri == 1) rr = (k.bcN == kPeriodic && r < 4 && r >= k.ny) ? r - k.ny : -1;
                if (rr < 0) continue;
                for (int ci = -1; ci < 2; ++ci) {
                    int cc = col;
                    if (ci == 0) cc = image(col, k.nx, k.bcE == kPeriodic);
                    if (ci == 1) cc = (k.bcE == kPeriodic && col < 4 && col >= k.nx) ? col - k.nx : -1;
                    if (cc < 0 || (ri < 0 && ci < 0)) continue;
                    put(rr, cc, e1, u1, v1);
                }
            }
        };
        images(row, ne.x, nhu.x, nhv.x);
        if (wr_y) images(row + kTileS, ne.y, nhu.y, nhv.y);
    }
}

// One stage of a tile whose corners and Coriolis rows lie in shared memory.
// fixed_ok: tile_load_fixed's answer.
template <bool RIM>
__device__ __forceinline__ void tile_stage(const StageArgs& a, const TileConst& tc, const TileIO& io, const float dt,
                                           const bool stage1, const TilePlace& t, const bool fixed_ok, TileSmem& sm) {
    const int lane = threadIdx.x & 31, w = warp_uniform((int)threadIdx.x >> 5);
    const float2 NZ = pb(a.neg_zero);
    // rim items: warps 0 .. 3 a row pair of the halo each, warp 4 the four halo columns of the tile's rows
    const bool rim_item = w < 5;
    const int rp = w < 2 ? w : (w < 4 ? kTileS + w : 2 + (lane >> 2));
    const int rq = w < 4 ? lane + 2 : ((lane & 2) ? kTileX + (lane & 3) : (lane & 3));
    const TileQ own = tile_load_q<RIM>(a, io, t, w + 2, lane + 2);
    TileQ edge{};
    if (rim_item) edge = tile_load_q<RIM>(a, io, t, rp, rq);
    const bool deep_floor = warp_uniform(__syncthreads_and(fixed_ok));     // also: the corners are in place
    float2 e, u, v;
    bool ok = tile_cell<RIM>(a, t, sm, w + 2, lane + 2, own, deep_floor, NZ, e, u, v);
    if (rim_item) {
        float2 e1, u1, v1;
        ok = tile_cell<RIM>(a, t, sm, rp, rq, edge, deep_floor, NZ, e1, u1, v1) && ok;
    }
    if (warp_uniform(__syncthreads_and(ok && deep_floor))) tile_phases<true, RIM>(a, tc, io, dt, stage1, t, sm, e, u, v);
    else tile_phases<false, RIM>(a, tc, io, dt, stage1, t, sm, e, u, v);
}

extern __shared__ __align__(16) unsigned char tile_smem_raw[];

__device__ __forceinline__ TileIO tile_io(const StageArgs& a) {
    return TileIO{a.eta_in, a.hu_in, a.hv_in, a.eta_out, a.hu_out, a.hv_out,
                  a.qn_eta, a.qn_hu, a.qn_hv, a.pin, a.pout, a.pqn};
}

// One stage, one tile per block.  Corners and Coriolis rows, which no stage
// writes, are read before the wait for the stage before (griddepcontrol.wait
// returns at once for a launch without the programmatic attribute; a stage
// launched with it follows another stage of the same call).
template <bool RIM>
__device__ __forceinline__ void tile_one(const StageArgs& a, const TileConst& tc, const TilePlace& t, TileSmem& sm) {
    const bool ok = tile_load_fixed<RIM>(a, t, sm);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    tile_stage<RIM>(a, tc, tile_io(a), a.dt, a.rk_step == 1, t, ok, sm);
}

__global__ void __launch_bounds__(kTileThreads, kTileBlocks)
    cdklm_tile_kernel(const __grid_constant__ StageArgs a, const __grid_constant__ TileConst tc) {
    TileSmem& sm = *reinterpret_cast<TileSmem*>(tile_smem_raw);
    const TilePlace t = tile_place(a.k, blockIdx.x, blockIdx.y);
    if (t.rim) tile_one<true>(a, tc, t, sm);
    else tile_one<false>(a, tc, t, sm);
}

// One batched stage: block i computes tile (member, column, row) of the packed
// list.  args holds two entries per member (stage 0: h0 -> h1, stage 1: h1 -> h0);
// dts holds the member's time step, read at launch so a captured graph picks
// up new values.
template <bool RIM>
__device__ __forceinline__ void tile_member(const StageArgs& a, const TileConst& tc, const float* dt,
                                            const TilePlace& t, TileSmem& sm) {
    const bool ok = tile_load_fixed<RIM>(a, t, sm);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    tile_stage<RIM>(a, tc, tile_io(a), __ldg(dt), a.rk_step == 1, t, ok, sm);
}

__global__ void __launch_bounds__(kTileThreads, kTileBlocks)
    cdklm_tile_batch_kernel(const StageArgs* __restrict__ args, const float* __restrict__ dts,
                            const TileConst* __restrict__ consts, const int4* __restrict__ tiles, const int rk_step) {
    TileSmem& sm = *reinterpret_cast<TileSmem*>(tile_smem_raw);
    const int4 tile = tiles[blockIdx.x];
    const StageArgs& a = args[2 * tile.x + rk_step];
    const TilePlace t = tile_place(a.k, tile.y, tile.z);
    if (warp_uniform(t.rim)) tile_member<true>(a, consts[tile.x], dts + tile.x, t, sm);
    else tile_member<false>(a, consts[tile.x], dts + tile.x, t, sm);
}

// n whole steps in one cooperative launch, one tile per block; a: the
// arguments of stage 0 (h0 -> h1), whose states stage 1 exchanges.  Every block takes
// part in every grid barrier, and a cooperative launch runs only when all its
// blocks are resident, so each wait ends.  States are read past L1
// (tile_load_q), which holds stale lines of what other blocks write between
// the barriers.
template <bool RIM>
__device__ __forceinline__ void tile_steps(const StageArgs& a, const TileConst& tc, const TilePlace& t, int n,
                                           TileSmem& sm) {
    const cooperative_groups::grid_group grid = cooperative_groups::this_grid();
    const bool ok = tile_load_fixed<RIM>(a, t, sm);
    float* const in[3] = {const_cast<float*>(a.eta_in), const_cast<float*>(a.hu_in), const_cast<float*>(a.hv_in)};
#pragma unroll 1
    for (int s = 0; s < 2 * n; ++s) {
        const bool stage1 = s & 1;
        TileIO io;
        io.e = stage1 ? a.eta_out : in[0]; io.hu = stage1 ? a.hu_out : in[1]; io.hv = stage1 ? a.hv_out : in[2];
        io.oe = stage1 ? in[0] : a.eta_out; io.ohu = stage1 ? in[1] : a.hu_out; io.ohv = stage1 ? in[2] : a.hv_out;
        io.ne = in[0]; io.nhu = in[1]; io.nhv = in[2];
        io.pin = stage1 ? a.pout : a.pin;
        io.pout = stage1 ? a.pin : a.pout;
        io.pn = a.pin;
        tile_stage<RIM>(a, tc, io, a.dt, stage1, t, ok, sm);
        if (s + 1 < 2 * n) grid.sync();
    }
}

__global__ void __launch_bounds__(kTileThreads, kTileStepsBlocks)
    cdklm_tile_steps_kernel(const __grid_constant__ StageArgs a, const __grid_constant__ TileConst tc, const int n) {
    TileSmem& sm = *reinterpret_cast<TileSmem*>(tile_smem_raw);
    const TilePlace t = tile_place(a.k, blockIdx.x, blockIdx.y);
    if (t.rim) tile_steps<true>(a, tc, t, n, sm);
    else tile_steps<false>(a, tc, t, n, sm);
}

}  // namespace go

// The fused RK2 step as a march of warp pairs up column strips.
//
// What bounds the step is instruction issue and the FP32 pipe (36 operations
// per byte of state), so this kernel is laid out to execute few instructions:
//   * a warp owns a strip of 64 columns (56 of them output, 4 halo columns on
//     each side for the two stages), two neighbouring columns per lane, and
//     marches north row by row.  Every operation on the two columns is one
//     paired instruction (f32x2.cuh).
//   * what a row needs from the rows below stays in registers: differences,
//     reconstructed face values and the flux through the south face are
//     computed once and handed to the next row, so no row is recomputed
//     within a run (the tile kernel recomputes 1.2 - 1.7 times and passes
//     every intermediate through shared memory between block barriers).
//     Values of the neighbouring columns come from warp shuffles.
//   * two warps share a strip: the first evaluates stage 1 and leaves Q* in
//     a ring of four rows in shared memory, the second marches three rows
//     behind with stage 2: row r of stage 1 completes row r - 2 of Q*, which is
//     read after the next barrier.  Each warp holds one stage's registers; they
//     meet at a barrier per row.  What both read is kept in rings of eight rows:
//     stage 2's oldest row lies five below the row of stage 1, the row that is
//     on its way two above it.
//   * rows of the inputs arrive two rows ahead in shared-memory rings
//     (cp.async), at column addresses that are fixed for a run, so periodic
//     images and wall mirrors cost nothing per row.
//   * common rows take no selects and few branches: a row whose faces are all
//     deeper than MarchConst::safe (no land, no shallow cell, no vanishing
//     wave speed) needs none of the scheme's rare cases.  Two warp votes
//     find the other rows, which a function of its own evaluates column by
//     column (march_row_general) from the same registers.
//
// The arithmetic is that of cdklm_tile.cuh, operation by operation and
// rounding by rounding (a value that several faces or terms of the tile
// kernel recompute is evaluated once here), so both give the same bits.
//
// Measured (256 members of 512 x 300, one step): 1.39 ms against 2.42 ms of
// the tile kernel; 96 members 0.566 against 0.945 ms, some 920 thread
// instructions per cell (warp instructions x 32) against 1,910, 62 % of the
// issue slots and 48 % of the FP32 pipe in use.  Eight strips per SM at 128
// registers a thread; six at 168 (1.72 ms) leave too few warps, ten at 96
// (1.75 ms) spill (128: none).
#pragma once

#include "cdklm_tile.cuh"

namespace goc {

constexpr int kMarchOut = 56;                 // output columns of a strip
constexpr int kMarchRows = 8;                 // rows of the unit a run is counted in
constexpr int kMarchRing = 8;                 // rows of the depth and Coriolis rings
constexpr int kMarchStage = 4;                // rows of the input and Q* rings
constexpr int kMarchThreads = 64;             // one warp per stage

// The buffers of one run.
struct MarchGrid {
    const float* e; const float* hu; const float* hv;     // Q^n
    float* e_out; float* hu_out; float* hv_out;           // Q^{n+1}
    const float* Hi; const float* Hm; const float* F;     // corner depths, cell means, Coriolis (or null)
    int pitch, hi_pitch, hm_pitch, f_pitch;               // floats
};

// Launch constants of the march: operands as pairs of equal halves.
struct MarchConst {
    float2 one, none, half, nhalf, quarter, two;
    float2 theta, theta_g, half_g, g, Vc, Uc, inv_2g, dx, dy, inv_dx, inv_dy, fb, rb;
    float safe;           // water depth above which a face is an ordinary wet one
    int general;          // parameters for which no row may take the short path
};

// Parameters of the member a strip belongs to.
struct MarchMember {
    GocCdklmParams p;
    StepConst k;
    MarchConst c;
};

// Shared memory of one strip: 32 lanes of two columns per row.
struct MarchSmem {
    float2 q[3][kMarchStage][32];      // Q^n as loaded (wall mirrors unsigned)
    float2 corner[kMarchStage][32];    // south-west corner depths as loaded
    float2 star[3][kMarchStage][32];   // Q*: the state after the first stage
    float2 qn[3][32];                  // Q^n of the output row
    float2 hm[kMarchRing][32];         // cell-mean depth
    float2 fc[kMarchRing][32];         // Coriolis f per cell, negated in ghost rows behind a wall
    float2 hc[kMarchRing][32];         // mean of each cell's corner depths, land corners at kDryFlag
    float2 hs[kMarchRing][32];         // depth of each cell's south face
    float2 hw[kMarchRing][32];         // depth of each cell's west face
    int2 col[3][32];                   // the lanes' columns: of the state, the cell fields and the corner depths
    int land[kMarchRing];              // corner row r or cell row r has land under the strip
    MarchGrid grid;
    MarchMember m;
    float nX, nY, wind_X, wind_Y;
    int x0;
};

// A face deeper than `safe` on both sides is wet, its cells are not shallow,
// and its wave speeds cannot vanish: ap - am >= 2 sqrt(g h) > flux_slope_eps.
// 0.1 m leaves the roundings of (eta + H) -+ t, evaluated in another order
// by the limiter's depth check, far below it.
__host__ __device__ inline MarchConst make_march_const(const GocCdklmParams& p, const StepConst& k) {
    auto two = [](float a) { return make_float2(a, a); };
    MarchConst m;
    m.one = k.one2; m.none = k.none2; m.half = k.half2; m.nhalf = two(-0.5f); m.quarter = k.quarter2;
    m.two = two(2.0f);
    m.theta = k.theta2; m.theta_g = k.theta_g2; m.half_g = k.half_g2; m.g = k.g2; m.Vc = k.Vc2; m.Uc = k.Uc2;
    m.inv_2g = two(k.inv_2g); m.dx = two(p.dx); m.dy = two(p.dy);
    m.inv_dx = two(k.inv_dx); m.inv_dy = two(k.inv_dy);
    m.fb = two(p.flux_balancer); m.rb = two(1.0f - p.flux_balancer);
    m.safe = fmaxf(fmaxf(0.1f, 2.0f * p.depth_cutoff),
                   fmaxf(1.01f * p.desing_eps, 0.3f * p.flux_slope_eps * p.flux_slope_eps / p.g));
    m.general = !(p.desing_eps > p.depth_cutoff) || p.one_dimensional;
    return m;
}

__device__ __forceinline__ float max3f(float a, float b, float c) { return fmaxf(fmaxf(a, b), c); }
__device__ __forceinline__ float min3f(float a, float b, float c) { return fminf(fminf(a, b), c); }
// minimum that keeps NaN, so that a NaN depth never passes for a safe one
__device__ __forceinline__ float min_nan(float a, float b) {
    float r;
    asm("min.NaN.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float min_nan(float2 a, float2 b) { return min_nan(min_nan(a.x, a.y), min_nan(b.x, b.y)); }

// Sums whose operands are no products: nothing to contract, no unit factor.
__device__ __forceinline__ float2 plain_add(float2 a, float2 b) {
    unsigned long long r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(b)));
    return unpack2(r);
}

__device__ __forceinline__ void cp_async4(void* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ float2 shfl_next_x(float2 own) {   // (own.y, next lane's x)
    return make_float2(own.y, __shfl_down_sync(0xffffffffu, own.x, 1));
}
__device__ __forceinline__ float2 shfl_prev_y(float2 own) {   // (previous lane's y, own.x)
    return make_float2(__shfl_up_sync(0xffffffffu, own.y, 1), own.x);
}

// Registers of a Runge-Kutta stage on its way up the strip, with L, C, U the
// rows j-1, j, j+1 when row j+1 arrives.
struct MarchState {
    float2 eL, uL, vL, eC, uC, vC;     // desingularised rows
    float2 fuL, fuC;                   // f times the east velocity
    float2 bu, bv, bK;                 // limiter differences across the face L|C
    float2 nE, nU, nV;                 // row L at its north face
    float2 eY;                         // row L: mean of the reconstructions at its south and north face
    float2 g0, g1, g2;                 // flux through the south face of row L
};

// Result of a row: tendencies of row L and the state the RK combination
// starts from.
struct MarchRhs {
    float2 fd0, r1, r2;                // d eta/dt = -fd0, d hu/dt = r1, d hv/dt = r2
    float2 e, hu, hv, Hm;
};

// Pairs of the fast path.
struct MarchOps {
    const MarchConst& c;
    __device__ __forceinline__ float2 add(float2 a, float2 b) const { return fma2(a, c.one, b); }
    __device__ __forceinline__ float2 sub(float2 a, float2 b) const { return fma2(b, c.none, a); }

    // minmod of both columns (minmod_raw; the sign of a zero result is free:
    // it is only ever added to or scaled)
    __device__ __forceinline__ float2 minmod(float2 a, float2 b, float2 d) const {
        const float2 hi = pr(fmaxf(min3f(a.x, b.x, d.x), 0.0f), fmaxf(min3f(a.y, b.y, d.y), 0.0f));
        const float2 lo = pr(fminf(max3f(a.x, b.x, d.x), 0.0f), fminf(max3f(a.y, b.y, d.y), 0.0f));
        return plain_add(hi, lo);
    }

    // Central-upwind flux (cdklm_flux) through two faces whose sides are all
    // deeper than `safe`: minus side (em, um, vm) of depth hm, plus side
    // (ep, up, vp) of depth hp; u normal, v transverse.
    __device__ __forceinline__ void flux(float2 em, float2 um, float2 vm, float2 hm, float2 ep, float2 up, float2 vp,
                                         float2 hp, float2& F0, float2& F1, float2& F2) const {
        const float2 gm = mul2(c.g, hm), gp = mul2(c.g, hp);
        const float2 cm = pr(sqrtf(gm.x), sqrtf(gm.y)), cp = pr(sqrtf(gp.x), sqrtf(gp.y));
        const float2 lm = sub(um, cm), lp = sub(up, cp), rm = add(um, cm), rp = add(up, cp);
        const float2 am = pr(min3f(lm.x, lp.x, 0.0f), min3f(lm.y, lp.y, 0.0f));
        const float2 ap = pr(max3f(rm.x, rp.x, 0.0f), max3f(rm.y, rp.y, 0.0f));
        const float2 d = sub(ap, am);
        const float2 inv = pr(1.0f / d.x, 1.0f / d.y);
        const float2 apam = mul2(ap, am);
        const float2 Fm0 = mul2(hm, um), Fp0 = mul2(hp, up);
        const float2 Fm2 = mul2(Fm0, vm), Fp2 = mul2(Fp0, vp);
        F0 = mul2(add(sub(mul2(ap, Fm0), mul2(am, Fp0)), mul2(apam, sub(ep, em))), inv);
        const float2 Fm1 = add(mul2(Fm0, um), mul2(mul2(c.half_g, hm), hm));
        const float2 Fp1 = add(mul2(Fp0, up), mul2(mul2(c.half_g, hp), hp));
        F1 = mul2(add(sub(mul2(ap, Fm1), mul2(am, Fp1)), mul2(apam, sub(Fp0, Fm0))), inv);
        const float2 up2 = mul2(c.fb, pr(um.x > -up.x ? Fm2.x : Fp2.x, um.y > -up.y ? Fm2.y : Fp2.y));
        const float2 s = sub(mul2(ap, Fm2), mul2(am, Fp2));
        const float2 h = sub(mul2(hp, vp), mul2(hm, vm));
        F2 = add(up2, mul2(c.rb, mul2(add(s, mul2(apam, h)), inv)));
    }
};

__device__ __forceinline__ bool any_lane(bool b) { return __any_sync(0xffffffffu, b) != 0; }
__device__ __forceinline__ unsigned march_ring(int r) { return (unsigned)(r & (kMarchRing - 1)) * 256u; }
__device__ __forceinline__ unsigned march_stage(int r) { return (unsigned)(r & (kMarchStage - 1)) * 256u; }
// the lane's pair of ring row `off` (byte offset of the row) of an array of MarchSmem
__device__ __forceinline__ float2& march_at(char* base, size_t array, unsigned off) {
    return *reinterpret_cast<float2*>(base + array + off);
}

// What a row takes and gives on the general path.
struct MarchCall {
    MarchState s;
    float2 e, hu, hv;       // the arriving row j+1 before desingularisation
    float2 su;
    MarchRhs R;
    int j, n;
};

// The tile kernel's limiters (minmod_raw2 of velocities, minmod_raw of balanced
// slopes) but for the sign of a zero.  MarchOps::minmod differs from them where
// an operand is NaN or infinite, so rows with such values take these.  A
// function of its own, so that the registers of its temporaries do not count in
// the marching loop (inlined: spills, 1.435 ms instead of 1.422, 256 members of
// 512 x 300; 1.419 without the test for such values).
static __device__ __noinline__ float2 march_limit(float2 b, float2 c, float2 f, bool velocity) {
    auto one = [&](float b, float c, float f) {
        const float m = fminf(fminf(fabsf(b), fabsf(c)), fabsf(f));
        const int B = __float_as_int(b);
        if (((B ^ __float_as_int(c)) | (B ^ __float_as_int(f))) >= 0) return copysignf(m, b);
        return velocity ? 0.0f * m : 0.0f;
    };
    return pr(one(b.x, c.x, f.x), one(b.y, c.y, f.y));
}

// Row j+1 of a stage arrives, the general way (`n` rows have arrived before
// it since the run began): any north angle, land, dry and shallow cells,
// one_dimensional.  Slopes of row j, flux through its south face, right-hand
// side of row j-1 (valid from n = 4 on), and the state one row further.
static __device__ __noinline__ void march_row_general(MarchSmem& S, MarchCall& call) {
    const GocCdklmParams& p = S.m.p;
    const StepConst& k = S.m.k;
    const MarchOps o{S.m.c};
    const int lane = threadIdx.x & 31, j = call.j, nx = p.nx, ny = p.ny;
    char* base = reinterpret_cast<char*>(&S) + lane * 8;
    const float nX = S.nX, nY = S.nY;
    const bool py = k.periodic_y;
    MarchState& s = call.s;
    constexpr size_t HS = offsetof(MarchSmem, hs), HW_ = offsetof(MarchSmem, hw), HC = offsetof(MarchSmem, hc),
                     FC = offsetof(MarchSmem, fc), HM = offsetof(MarchSmem, hm);
    const unsigned oL = march_ring(j - 1), oC = march_ring(j), oU = march_ring(j + 1);
    auto flux_face = [&](float em, float um, float vm, float ep, float up, float vp, float Hf, bool dm, bool dp,
                         float& F0, float& F1, float& F2) {
        const bool still = cdklm_flux(p, k, em, um, vm, ep, up, vp, Hf, F0, F1, F2);
        if (still) { F0 = 0.f; F1 = 0.f; F2 = 0.f; }
        if (dm || dp) {
            F0 = 0.f; F2 = 0.f;
            F1 = (dm && dp) ? 0.f : dm ? k.half_g * (ep + Hf) * (ep + Hf) : k.half_g * (em + Hf) * (em + Hf);
        }
    };
    // the depth check of one cell's limited balanced slope K; Ha / Hb: depths
    // of its lower and upper face; check: the Coriolis term with the sign
    // with which it is added to K
    auto checked = [&](float K, float e, float Ha, float Hb, float check) {
        const float t = (K + check) * k.inv_2g;
        const float ha = e + Ha - t, hb = e + Hb + t;
        K = (ha > 0.0f) ? K : -check + k.two_g * (e + Ha);
        K = (hb > 0.0f) ? K : -check - k.two_g * (e + Hb);
        return K;
    };

    float2 eU, uU, vU;
    {
        const float2 Hm = march_at(base, HM, oU);
        desingularize_cell(p, call.e.x, call.hu.x, call.hv.x, Hm.x, eU.x, uU.x, vU.x);
        desingularize_cell(p, call.e.y, call.hu.y, call.hv.y, Hm.y, eU.y, uU.y, vU.y);
    }
    // whether the rows hold a value that is not finite
    const float2 sum = plain_add(plain_add(plain_add(s.eL, s.uL), plain_add(s.vL, s.eC)),
                                 plain_add(plain_add(s.uC, s.vC), plain_add(plain_add(eU, uU), vU)));
    const bool wild = any_lane(!(fabsf(sum.x) + fabsf(sum.y) < INFINITY));
    const bool ghostU = !py && (j + 1 < 2 || j + 1 >= ny + 2), ghostC = !py && (j < 2 || j >= ny + 2);
    const float sU_ = ghostU ? -1.0f : 1.0f, sC_ = ghostC ? -1.0f : 1.0f;
    // Coriolis f without the ghost rows' sign, which acts on u alone
    const float2 fU = mul2(march_at(base, FC, oU), pr(sU_)), fC = mul2(march_at(base, FC, oC), pr(sC_));
    const float2 fuU = mul2(o.add(mul2(pr(nY), mul2(uU, pr(sU_))), mul2(pr(-nX), vU)), fU);
    // ---- y slopes of row C ----
    const float2 du = mul2(o.sub(uU, s.uC), o.c.theta), dv = mul2(o.sub(vU, s.vC), o.c.theta);
    const float2 dK = mul2(o.c.theta_g, o.add(o.sub(eU, s.eC), mul2(o.c.Uc, o.add(s.fuC, fuU))));
    const float2 cu = mul2(o.sub(uU, s.uL), o.c.half), cv = mul2(o.sub(vU, s.vL), o.c.half);
    const float2 cK = mul2(o.c.half_g, o.add(o.sub(eU, s.eL), mul2(o.c.Uc, o.add(fma2(s.fuC, o.c.two, fuU), s.fuL))));
    float2 mu = o.minmod(s.bu, cu, du), mv = o.minmod(s.bv, cv, dv), Ly = o.minmod(s.bK, cK, dK);
    if (wild) {
        mu = march_limit(s.bu, cu, du, true);
        mv = march_limit(s.bv, cv, dv, true);
        Ly = march_limit(s.bK, cK, dK, false);
    }
    const float2 HsC = march_at(base, HS, oC), HsU = march_at(base, HS, oU);
    float2 tY, sE, nE;
    {
        const float ua_sign = (p.bc_south == 1 && j < 2) || (p.bc_north == 1 && j > ny + 2) ? -1.0f : 1.0f;
        auto cell = [&](float L, float e, float u, float v, float f, float Hs, float Hn, float& t, float& es, float& en) {
            L = checked(L, e, Hs, Hn, -(p.dy * f * (ua_sign * u)));
            const float tf = (L - p.dy * f * ((sC_ * u) * nY + v * (-nX))) * k.inv_2g;
            t = (L - p.dy * f * u) * k.inv_2g;      // as the sources see it
            es = fmaxf(-Hs, e - tf);
            en = fmaxf(-Hn, e + tf);
        };
        cell(Ly.x, s.eC.x, s.uC.x, s.vC.x, fC.x, HsC.x, HsU.x, tY.x, sE.x, nE.x);
        cell(Ly.y, s.eC.y, s.uC.y, s.vC.y, fC.y, HsC.y, HsU.y, tY.y, sE.y, nE.y);
    }
    const float2 sU = fma2(mu, o.c.nhalf, s.uC), sV = fma2(mv, o.c.nhalf, s.vC);
    const float2 nU = fma2(mu, o.c.half, s.uC), nV = fma2(mv, o.c.half, s.vC);
    // ---- flux through the face L|C (u and v swap roles) ----
    float2 g0, g1, g2;
    flux_face(s.nE.x, s.nV.x, s.nU.x, sE.x, sV.x, sU.x, HsC.x, s.eL.x == kDryFlag, s.eC.x == kDryFlag, g0.x, g2.x, g1.x);
    flux_face(s.nE.y, s.nV.y, s.nU.y, sE.y, sV.y, sU.y, HsC.y, s.eL.y == kDryFlag, s.eC.y == kDryFlag, g0.y, g2.y, g1.y);

    if (call.n >= 4) {
        // ---- x direction and right-hand side of row L ----
        const float2 e = s.eL, u = s.uL, v = s.vL, su = call.su, f = march_at(base, FC, oL);
        const float2 vs = mul2(v, su);
        const float2 fv = mul2(o.add(mul2(pr(nX), u), mul2(pr(nY), vs)), f);
        const float2 eM = shfl_prev_y(e), eP = shfl_next_x(e);
        const float2 uM = shfl_prev_y(u), uP = shfl_next_x(u);
        const float2 vM = shfl_prev_y(v), vP = shfl_next_x(v);
        const float2 fM = shfl_prev_y(fv), fP = shfl_next_x(fv);
        const float2 th = o.c.theta, hf = o.c.half;
        const float2 bU = mul2(o.sub(u, uM), th), cU = mul2(o.sub(uP, uM), hf), dU = mul2(o.sub(uP, u), th);
        const float2 bV = mul2(o.sub(v, vM), th), cV = mul2(o.sub(vP, vM), hf), dV = mul2(o.sub(vP, v), th);
        float2 xu = o.minmod(bU, cU, dU), xv = o.minmod(bV, cV, dV);
        const float2 bK = mul2(o.c.theta_g, o.sub(o.sub(e, eM), mul2(o.c.Vc, o.add(fv, fM))));
        const float2 eK = mul2(o.c.theta_g, o.sub(o.sub(eP, e), mul2(o.c.Vc, o.add(fv, fP))));
        const float2 xK = mul2(o.c.half_g, o.sub(o.sub(eP, eM), mul2(o.c.Vc, o.add(fma2(fv, o.c.two, fP), fM))));
        float2 Kx = o.minmod(bK, xK, eK);
        if (wild) {
            xu = march_limit(bU, cU, dU, true);
            xv = march_limit(bV, cV, dV, true);
            Kx = march_limit(bK, xK, eK, false);
        }
        const float2 HW = march_at(base, HW_, oL), HE = shfl_next_x(HW);
        float2 tX, wE, xE;
        auto cell = [&](int q, float K, float ee, float uu, float vv, float sgn, float ff, float Ha, float Hb, float& t,
                        float& ew, float& en) {
            // gx < 2 or > nx + 2: behind a wall (columns carry the sign too,
            // but the check sees the ghost column nx + 2 unmirrored)
            const int gx = S.x0 + 2 * lane + q;
            const float va = (p.bc_west == 1 && gx < 2) || (p.bc_east == 1 && gx > nx + 2) ? -vv : vv;
            K = checked(K, ee, Ha, Hb, p.dx * ff * va);
            const float tf = (K + p.dx * ff * (uu * nX + (sgn * vv) * nY)) * k.inv_2g;
            t = (K + p.dx * ff * vv) * k.inv_2g;        // as the sources see it
            ew = fmaxf(-Ha, ee - tf);
            en = fmaxf(-Hb, ee + tf);
        };
        cell(0, Kx.x, e.x, u.x, v.x, su.x, f.x, HW.x, HE.x, tX.x, wE.x, xE.x);
        cell(1, Kx.y, e.y, u.y, v.y, su.y, f.y, HW.y, HE.y, tX.y, wE.y, xE.y);
        const float2 wU = fma2(xu, o.c.nhalf, u), wV = fma2(xv, o.c.nhalf, v);
        const float2 xU = fma2(xu, o.c.half, u), xV = fma2(xv, o.c.half, v);
        const float2 pE = shfl_next_x(wE), pU = shfl_next_x(wU), pV = shfl_next_x(wV);
        const bool d0 = e.x == kDryFlag, d1 = e.y == kDryFlag, d2 = eP.y == kDryFlag;
        float2 F0, F1, F2;
        flux_face(xE.x, xU.x, xV.x, pE.x, pU.x, pV.x, HE.x, d0, d1, F0.x, F1.x, F2.x);
        flux_face(xE.y, xU.y, xV.y, pE.y, pU.y, pV.y, HE.y, d1, d2, F0.y, F1.y, F2.y);
        float2 fd0 = mul2(o.sub(F0, shfl_prev_y(F0)), o.c.inv_dx);
        float2 fd1 = mul2(o.sub(F1, shfl_prev_y(F1)), o.c.inv_dx);
        float2 fd2 = mul2(o.sub(F2, shfl_prev_y(F2)), o.c.inv_dx);
        if (!p.one_dimensional) {
            fd0 = o.add(fd0, mul2(o.sub(g0, s.g0), o.c.inv_dy));
            fd1 = o.add(fd1, mul2(o.sub(g1, s.g1), o.c.inv_dy));
            fd2 = o.add(fd2, mul2(o.sub(g2, s.g2), o.c.inv_dy));
        }
        // the tile kernel's cell_state and source terms, one column
        const float2 Hm = march_at(base, HC, oL), hsum = o.add(e, Hm);
        const float2 HS0 = march_at(base, HS, oL);
        auto source = [&](float ee, float uu, float vv, float ff, float H, float hs, float tx, float eYm, float dHx,
                          float dHy, float fl1, float fl2, float& hu, float& hv, float& r1, float& r2) {
            hu = hs > p.depth_cutoff ? uu * hs : 0.0f;
            hv = hs > p.depth_cutoff ? vv * hs : 0.0f;
            const float eX = nY, eY = -nX, upx = -nX, upy = nY;
            const float hu_e = hu * eX + hv * eY, hv_n = hu * nX + hv * nY;
            const float hu_ec = ff * hv_n, hv_nc = -ff * hu_e;
            const float hu_cor = upy * hu_ec + (-upx) * hv_nc, hv_cor = upx * hu_ec + upy * hv_nc;
            const float eXm = 0.5f * ((ee - tx) + (ee + tx));
            float st1 = S.wind_X + hu_cor + p.g * (eXm + H) * dHx * k.inv_dx;
            float st2 = S.wind_Y + hv_cor + p.g * (eYm + H) * dHy * k.inv_dy;
            if (!(hs >= p.depth_cutoff && ee != kDryFlag)) { st1 = 0.0f; st2 = 0.0f; }
            r1 = -fl1 + st1;
            r2 = -fl2 + st2;
        };
        MarchRhs& R = call.R;
        source(e.x, u.x, v.x, f.x, Hm.x, hsum.x, tX.x, s.eY.x, HE.x - HW.x, HsC.x - HS0.x, fd1.x, fd2.x, R.hu.x, R.hv.x,
               R.r1.x, R.r2.x);
        source(e.y, u.y, v.y, f.y, Hm.y, hsum.y, tX.y, s.eY.y, HE.y - HW.y, HsC.y - HS0.y, fd1.y, fd2.y, R.hu.y, R.hv.y,
               R.r1.y, R.r2.y);
        R.fd0 = fd0;
        R.Hm = Hm;
        R.e = e;
    }
    s.bu = du; s.bv = dv; s.bK = dK;
    s.nE = nE; s.nU = nU; s.nV = nV;
    s.eY = mul2(o.c.half, o.add(o.add(s.eC, tY), o.sub(s.eC, tY)));
    s.g0 = g0; s.g1 = g1; s.g2 = g2;
    s.fuL = s.fuC; s.fuC = fuU;
    s.eL = s.eC; s.uL = s.uC; s.vL = s.vC;
    s.eC = eU; s.uC = uU; s.vC = vU;
}

// The strip's two warps (the whole CTA) meet.
__device__ __forceinline__ void march_barrier() {
    asm volatile("bar.sync 0, %0;" ::"n"(kMarchThreads) : "memory");
}

// The periodic ghost images of a cell (store_with_images without the cell
// itself).
__device__ __forceinline__ void store_images(const GocCdklmParams& p, const StepConst& k, const MarchGrid& G, int gx,
                                             int gy, float e, float hu, float hv) {
    const int ix = !k.periodic_x ? -1 : gx < 4 ? gx + p.nx : gx >= p.nx ? gx - p.nx : -1;
    const int iy = !k.periodic_y ? -1 : gy < 4 ? gy + p.ny : gy >= p.ny ? gy - p.ny : -1;
    auto put = [&](int x, int y) {
        const size_t o = (size_t)y * G.pitch + x;
        G.e_out[o] = e; G.hu_out[o] = hu; G.hv_out[o] = hv;
    };
    if (ix >= 0) put(ix, gy);
    if (iy >= 0) put(gx, iy);
    if (ix >= 0 && iy >= 0) put(ix, iy);
}

// Semi-implicit friction coefficient (the tile kernel's friction).
__device__ __forceinline__ float march_friction(const GocCdklmParams& p, float dt, float hs, float hu, float hv) {
    if (hs < p.desing_eps) {
        const float u = desing(hs, hu, p.desing_eps), v = desing(hs, hv, p.desing_eps);
        return dt * p.r * desing(hs, sqrtf(u * u + v * v), p.desing_eps);
    }
    const float u = hu / hs, v = hv / hs;
    return dt * p.r * sqrtf(u * u + v * v) / hs;
}

// Output rows [row0, row1) of the strip's columns (row0 = 2 or at least 4):
// one RK2 step of length dt.
// p, k, c: the scalar parameters, in the kernel's parameter space or equal to
// S.m; pm: the member's own (textures).  Called by the two warps of a strip
// together, with S.grid and S.m set and a barrier since.
__device__ __forceinline__ void march_run(const GocCdklmParams& p, const GocCdklmParams& pm, const StepConst& k,
                                          const MarchConst& c, MarchSmem& S, float dt, int strip, int row0,
                                          int row1) {
    const MarchGrid& G = S.grid;
    const int lane = threadIdx.x & 31;
    // stage 2; broadcast so that what depends on it is known to be the same in the warp
    const bool second = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0) != 0;
    const int nx = p.nx, ny = p.ny;
    const bool px = k.periodic_x, py = k.periodic_y;
    const int x0 = 2 + strip * kMarchOut - 4, gx0 = x0 + 2 * lane;
    char* const base = reinterpret_cast<char*>(&S) + lane * 8;
    const MarchOps o{c};
    constexpr size_t ST = offsetof(MarchSmem, star), Q = offsetof(MarchSmem, q), HS = offsetof(MarchSmem, hs),
                     HW_ = offsetof(MarchSmem, hw), HC = offsetof(MarchSmem, hc), HM = offsetof(MarchSmem, hm),
                     FC = offsetof(MarchSmem, fc), CO = offsetof(MarchSmem, corner), QN = offsetof(MarchSmem, qn);
    constexpr size_t P = sizeof(float2) * 32 * kMarchStage;
    auto at = [&](size_t array, unsigned off) -> float2& { return march_at(base, array, off); };

    const float angle = __ldg(pm.angle), wt = pm.wind_t;
    const float nX = __sinf(angle), nY = __cosf(angle);
    const float wind_X = pm.wind_stress_factor * (wt * __ldg(pm.wind_x_next) + (1.0f - wt) * __ldg(pm.wind_x_cur));
    const float wind_Y = pm.wind_stress_factor * (wt * __ldg(pm.wind_y_next) + (1.0f - wt) * __ldg(pm.wind_y_cur));
    const bool general = c.general || nX != 0.0f || nY != 1.0f;
    const bool east = !px && x0 + 63 >= nx + 2;          // holds the ghost column nx + 2 behind an east wall
    const bool wall_x = !px && (x0 < 2 || east);
    const float f0 = G.F ? 0.0f : __ldg(pm.coriolis_f);  // one Coriolis value
    if (threadIdx.x == 0) {
        S.nX = nX; S.nY = nY; S.wind_X = wind_X; S.wind_Y = wind_Y; S.x0 = x0;
    }

    // the lane's two columns: of the state (periodic images wrapped, wall
    // mirrors folded back), of the cell fields and of the corner depths
    bool pairs;
    float2 su;                                           // -1 in ghost columns behind a wall, else 1
    {
        int cq[2], ch[2], ca[2];
        float sg[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int gx = gx0 + i;
            sg[i] = 1.0f;
            if (px) {
                cq[i] = ch[i] = ca[i] = wrap_interior(gx, nx);
            } else {
                int mx = gx;
                if (gx == nx + 2 || gx == nx + 3) { mx = 2 * nx + 3 - gx; sg[i] = -1.0f; }
                if (gx == 0 || gx == 1) { mx = 3 - gx; sg[i] = -1.0f; }
                cq[i] = clampi(mx, 0, nx + 3);
                ch[i] = clampi(gx, 0, nx + 3);
                ca[i] = clampi(gx, 0, nx + 4);
            }
        }
        su = pr(sg[0], sg[1]);
        // pairs of adjacent columns on 8-byte boundaries load as one
        const bool adj = cq[1] == cq[0] + 1 && ch[1] == ch[0] + 1 && (cq[0] & 1) == 0 && (ch[0] & 1) == 0;
        pairs = __all_sync(0xffffffffu, adj) &&
                (((uintptr_t)G.e | (uintptr_t)G.hu | (uintptr_t)G.hv | (uintptr_t)G.Hm | (uintptr_t)G.F) & 7u) == 0 &&
                ((G.pitch | G.hm_pitch | (G.F ? G.f_pitch : 0)) & 1) == 0;
        if (!second) {     // read by the same lanes only
            S.col[0][lane] = make_int2(cq[0], cq[1]);
            S.col[1][lane] = make_int2(ch[0], ch[1]);
            S.col[2][lane] = make_int2(ca[0], ca[1]);
        }
    }
    // output columns of the lane
    const bool mine = lane >= 2 && lane < 30;
    const bool o0 = mine && gx0 < nx + 2, o1 = mine && gx0 + 1 < nx + 2;
    const bool wide = pairs && (((uintptr_t)G.e_out | (uintptr_t)G.hu_out | (uintptr_t)G.hv_out) & 7u) == 0;
    const bool x_images = px && (x0 < 4 || x0 + 63 >= nx);

    // rows: inputs [a0, a1], second stage [b0, b1]; row r of stage 1 yields
    // Q* of row r - 2, row r of stage 2 the output row r - 2.  Stage 2 takes a
    // row three behind stage 1, whose Q* was written before the last barrier;
    // at a south wall it starts with rows 3 and 2 mirrored, and stage 1 waits
    // three rows while it catches up.
    const int a0 = py ? row0 - 4 : max(row0 - 4, 0), a1 = py ? row1 + 3 : min(row1 + 3, ny + 3);
    const int b0 = row0 - 2, b1 = row1 + 1;
    const bool south = !py && b0 < 2;
    const int delay = south ? 6 : b0 - a0 + 3;
    const unsigned in = second ? (unsigned)ST : (unsigned)Q;
    const float2 d2 = pr(dt);

    auto issue = [&](int r) {
        const int rh = py ? wrap_interior(r, ny) : clampi(r, 0, ny + 3);
        const int ra = py ? rh : clampi(r, 0, ny + 4);
        int rq = rh;
        if (!py) {
            if (r == ny + 2 || r == ny + 3) rq = clampi(2 * ny + 3 - r, 0, ny + 3);
            if (r == 0 || r == 1) rq = 3 - r;
        }
        const unsigned s4 = march_stage(r), s8 = march_ring(r);
        const size_t oq = (size_t)rq * G.pitch, oh = (size_t)rh * G.hm_pitch;
        const float* A = G.Hi + (size_t)ra * G.hi_pitch;
        const float* F = G.F;
        const int2 cq = S.col[0][lane], ch = S.col[1][lane], ca = S.col[2][lane];
        float* d0 = &at(Q, s4).x;
        float* da = &at(CO, s4).x;
        float* dh = &at(HM, s8).x;
        float* df = &at(FC, s8).x;
        if (pairs) {
            cp_async8(d0, G.e + oq + cq.x);
            cp_async8(d0 + P / 4, G.hu + oq + cq.x);
            cp_async8(d0 + P / 2, G.hv + oq + cq.x);
            cp_async8(dh, G.Hm + oh + ch.x);
            if (F) cp_async8(df, F + (size_t)rh * G.f_pitch + ch.x);
        } else {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int q = i ? cq.y : cq.x, h = i ? ch.y : ch.x;
                cp_async4(d0 + i, G.e + oq + q);
                cp_async4(d0 + P / 4 + i, G.hu + oq + q);
                cp_async4(d0 + P / 2 + i, G.hv + oq + q);
                cp_async4(dh + i, G.Hm + oh + h);
                if (F) cp_async4(df + i, F + (size_t)rh * G.f_pitch + h);
            }
        }
        cp_async4(da, A + ca.x);
        cp_async4(da + 1, A + ca.y);
    };
    if (!second) {
        if (!G.F)
            for (int i = 0; i < kMarchRing; ++i) at(FC, i * 256u) = pr(f0);
        issue(a0);
        cp_async_commit();
        issue(a0 + 1);
        cp_async_commit();
    }
    MarchState s{};
    unsigned hist = 0;                                   // bit i: row r - i has land under the strip
    const int r0 = second ? b0 : a0, r1 = second ? b1 : a1;
    int r = r0, idle = second ? delay : 0;
    for (int t = delay + b1 - b0 + 1; t > 0; --t) {
        if (idle > 0 || r > r1) {
            --idle;
            march_barrier();
            continue;
        }
        const int n = r - r0;
        const unsigned oU = march_ring(r), oC = march_ring(r - 1), oL = march_ring(r - 2);
        const size_t og = (size_t)(r - 2) * G.pitch + gx0;
        unsigned s4 = march_stage(r);
        bool flip = false, lands = false;
        const bool ghost_row = !py && (unsigned)(r - 2) >= (unsigned)ny;     // beyond a wall
        hist = hist << 1 | (unsigned)general;
        if (second) {
            // input row Q*, wall mirrors folded back, and Q^n of the output row
            if (__builtin_expect(ghost_row, 0)) {
                s4 = march_stage(r < 2 ? 3 - r : 2 * ny + 3 - r);
                flip = true;
            }
            if (n >= 4) {
                float* d0 = &at(QN, 0).x;
                if (wide) {
                    if (o0) {
                        cp_async8(d0, G.e + og);
                        cp_async8(d0 + 64, G.hu + og);
                        cp_async8(d0 + 128, G.hv + og);
                    }
                } else {
                    if (o0) { cp_async4(d0, G.e + og); cp_async4(d0 + 64, G.hu + og); cp_async4(d0 + 128, G.hv + og); }
                    if (o1) { cp_async4(d0 + 1, G.e + og + 1); cp_async4(d0 + 65, G.hu + og + 1); cp_async4(d0 + 129, G.hv + og + 1); }
                }
            }
            hist |= (unsigned)S.land[r & (kMarchRing - 1)];
        } else {
            if (r + 2 <= a1) issue(r + 2);
            cp_async_commit();
            cp_async_wait<2>();
            if (__builtin_expect(ghost_row, 0)) {
                flip = true;
                float2& f = at(FC, oU);
                f = G.F ? pr(-f.x, -f.y) : pr(-f0);
            } else if (__builtin_expect(!py && (r == 8 || r == 9), 0)) {
                if (!G.F) at(FC, oU) = pr(f0);           // the ring rows of the ghost rows 0 and 1
            }
            const float2 A = at(CO, s4), Hmb = at(HM, oU);
            lands = fabsf(A.x - p.land_value) < kDryEps || fabsf(A.y - p.land_value) < kDryEps ||
                    fabsf(Hmb.x - p.land_value) <= kDryEps || fabsf(Hmb.y - p.land_value) <= kDryEps;
        }
        // ---- row U arrives ----
        const float2 eU = at(in, s4);
        float2 hu = at(in + P, s4), hv = at(in + 2 * P, s4);
        if (__builtin_expect(wall_x, 0)) hu = second ? hu : mul2(hu, su);   // Q* is mirrored when written
        if (__builtin_expect(flip, 0)) hv = pr(-hv.x, -hv.y);
        const float2 h = plain_add(eU, at(HM, oU));
        const float2 ih = pr(1.0f / h.x, 1.0f / h.y);
        const float2 uU = mul2(hu, ih), vU = mul2(hv, ih);
        // h + 0 (hu^2 + hv^2): NaN where a momentum is not finite, or so large that
        // a velocity might not be
        const float2 hf = fma2(fma2(hu, hu, mul2(hv, hv)), pr(0.0f), h);
        // eta of a wet cell at the value that marks dry ones, which the scheme
        // takes for one
        const bool flag = eU.x == kDryFlag || eU.y == kDryFlag;
        bool bad = lands || flag || !(min_nan(hf.x, hf.y) >= p.desing_eps);

        // ---- balanced x slope of row L and its depth check ----
        float2 wE, xE;
        if (n >= 4) {
            const float2 vs = mul2(s.vL, su), f = at(FC, oL), fv = mul2(vs, f);
            const float2 eM = shfl_prev_y(s.eL), eP = shfl_next_x(s.eL);
            const float2 fM = shfl_prev_y(fv), fP = shfl_next_x(fv);
            const float2 bK = mul2(c.theta_g, o.sub(o.sub(s.eL, eM), mul2(c.Vc, o.add(fv, fM))));
            const float2 dK = mul2(c.theta_g, o.sub(o.sub(eP, s.eL), mul2(c.Vc, o.add(fv, fP))));
            const float2 cK = mul2(c.half_g, o.sub(o.sub(eP, eM), mul2(c.Vc, o.add(fma2(fv, c.two, fP), fM))));
            const float2 Kx = o.minmod(bK, cK, dK);
            const float2 dxf = mul2(c.dx, f);
            const float2 HW = at(HW_, oL), HE = shfl_next_x(HW);
            const float2 tX = mul2(o.add(Kx, mul2(dxf, vs)), c.inv_2g);
            wE = o.sub(s.eL, tX);
            xE = o.add(s.eL, tX);
            const float2 hsum = plain_add(s.eL, at(HC, oL));
            bool bad_x = !(min_nan(min_nan(o.add(wE, HW), o.add(xE, HE)), min_nan(hsum.x, hsum.y)) > c.safe);
            if (__builtin_expect(east, 0)) {
                // the ghost column beyond an east wall: its depth check takes
                // the velocity unmirrored
                auto dry = [&](int q, float K, float df, float vv, float ee, float Ha, float Hb) {
                    const float t_ = (K + df * vv) * k.inv_2g;
                    return gx0 + q == nx + 2 && !(ee + Ha - t_ > 0.0f && ee + Hb + t_ > 0.0f);
                };
                bad_x = bad_x || dry(0, Kx.x, dxf.x, s.vL.x, s.eL.x, HW.x, HE.x) ||
                        dry(1, Kx.y, dxf.y, s.vL.y, s.eL.y, HW.y, HE.y);
            }
            bad = bad || bad_x;
        }
        bool slow = any_lane(bad);
        // a row with land, such a value or a momentum that is not finite takes
        // the general path until it has left the pipeline
        if (__builtin_expect(slow, 0) && any_lane(lands || flag || hf.x != hf.x || hf.y != hf.y)) hist |= 1u;
        if (!second) {
            // the depths that row U completes
            float2 A = at(CO, s4);
            if (__builtin_expect(slow, 0)) {
                const bool lx = fabsf(A.x - p.land_value) < kDryEps, ly = fabsf(A.y - p.land_value) < kDryEps;
                if (lx) A.x = kDryFlag;
                if (ly) A.y = kDryFlag;
                at(CO, s4) = A;
            }
            const float2 B = shfl_next_x(A), Ap = at(CO, march_stage(r - 1)), Bp = shfl_next_x(Ap);
            const float2 AA = plain_add(Ap, A);
            at(HS, oU) = mul2(c.half, plain_add(A, B));
            at(HW_, oC) = mul2(c.half, AA);
            at(HC, oC) = mul2(c.quarter, plain_add(plain_add(AA, Bp), B));
            if (lane == 0) S.land[r & (kMarchRing - 1)] = (int)(hist & 1u);
        }
        slow = slow || (hist & 7u) != 0 || (ghost_row && r == ny + 3);
        MarchRhs R;
        if (__builtin_expect(!slow, 1)) {
            // ---- y slopes of row C ----
            const float2 fuU = mul2(uU, at(FC, oU));
            const float2 du = mul2(o.sub(uU, s.uC), c.theta), dv = mul2(o.sub(vU, s.vC), c.theta);
            const float2 dK = mul2(c.theta_g, o.add(o.sub(eU, s.eC), mul2(c.Uc, o.add(s.fuC, fuU))));
            const float2 cK = mul2(c.half_g, o.add(o.sub(eU, s.eL), mul2(c.Uc, o.add(fma2(s.fuC, c.two, fuU), s.fuL))));
            const float2 Ly = o.minmod(s.bK, cK, dK);
            const float2 HsC = at(HS, oC);
            const float2 tY = mul2(o.sub(Ly, mul2(mul2(c.dy, at(FC, oC)), s.uC)), c.inv_2g);
            const float2 sE = o.sub(s.eC, tY), nE = o.add(s.eC, tY);
            const float2 hp = o.add(sE, HsC), hl = o.add(s.nE, HsC);
            const bool bad_y = !(min_nan(min_nan(hp, o.add(nE, at(HS, oU))), min_nan(hl.x, hl.y)) > c.safe);
            if (__builtin_expect(any_lane(bad_y && n >= 2), 0)) {
                slow = true;
            } else {
                const float2 cu = mul2(o.sub(uU, s.uL), c.half), cv = mul2(o.sub(vU, s.vL), c.half);
                const float2 mu = o.minmod(s.bu, cu, du), mv = o.minmod(s.bv, cv, dv);
                const float2 sU = fma2(mu, c.nhalf, s.uC), sV = fma2(mv, c.nhalf, s.vC);
                // ---- flux through the face L|C (u and v swap roles) ----
                float2 g0, g1, g2;
                o.flux(s.nE, s.nV, s.nU, hl, sE, sV, sU, hp, g0, g2, g1);
                R.fd0 = mul2(o.sub(g0, s.g0), c.inv_dy);
                const float2 fy1 = mul2(o.sub(g1, s.g1), c.inv_dy), fy2 = mul2(o.sub(g2, s.g2), c.inv_dy);
                R.Hm = at(HC, oL);
                const float2 bathy = mul2(mul2(mul2(c.g, o.add(s.eY, R.Hm)), o.sub(HsC, at(HS, oL))), c.inv_dy);
                s.nU = fma2(mu, c.half, s.uC);
                s.nV = fma2(mv, c.half, s.vC);
                s.nE = nE;
                s.eY = mul2(c.half, o.add(nE, sE));
                s.bu = du; s.bv = dv; s.bK = dK;
                s.g0 = g0; s.g1 = g1; s.g2 = g2;
                s.fuL = s.fuC; s.fuC = fuU;
                // ---- x slopes and fluxes, right-hand side of row L ----
                if (n >= 4) {
                    const float2 u = s.uL, v = s.vL;
                    const float2 uM = shfl_prev_y(u), uP = shfl_next_x(u);
                    const float2 vM = shfl_prev_y(v), vP = shfl_next_x(v);
                    const float2 xu = o.minmod(mul2(o.sub(u, uM), c.theta), mul2(o.sub(uP, uM), c.half), mul2(o.sub(uP, u), c.theta));
                    const float2 xv = o.minmod(mul2(o.sub(v, vM), c.theta), mul2(o.sub(vP, vM), c.half), mul2(o.sub(vP, v), c.theta));
                    const float2 HW = at(HW_, oL), HE = shfl_next_x(HW);
                    const float2 pU = shfl_next_x(fma2(xu, c.nhalf, u)), pV = shfl_next_x(fma2(xv, c.nhalf, v));
                    const float2 pE = shfl_next_x(wE);
                    float2 F0, F1, F2;
                    o.flux(xE, fma2(xu, c.half, u), fma2(xv, c.half, v), o.add(xE, HE), pE, pU, pV, o.add(pE, HE), F0, F1, F2);
                    R.fd0 = o.add(mul2(o.sub(F0, shfl_prev_y(F0)), c.inv_dx), R.fd0);
                    const float2 fd1 = o.add(mul2(o.sub(F1, shfl_prev_y(F1)), c.inv_dx), fy1);
                    const float2 fd2 = o.add(mul2(o.sub(F2, shfl_prev_y(F2)), c.inv_dx), fy2);
                    const float2 hsum = plain_add(s.eL, R.Hm), f = at(FC, oL);
                    R.e = s.eL;
                    R.hu = mul2(u, hsum);
                    R.hv = mul2(v, hsum);
                    const float2 eX = mul2(c.half, o.add(wE, xE));
                    const float2 bathx = mul2(mul2(mul2(c.g, o.add(eX, R.Hm)), o.sub(HE, HW)), c.inv_dx);
                    R.r1 = o.sub(o.add(o.add(pr(wind_X), mul2(f, R.hv)), bathx), fd1);
                    R.r2 = o.sub(o.add(o.sub(pr(wind_Y), mul2(f, R.hu)), bathy), fd2);
                }
                s.eL = s.eC; s.uL = s.uC; s.vL = s.vC;
                s.eC = eU; s.uC = uU; s.vC = vU;
            }
        }
        if (__builtin_expect(slow, 0)) {
            MarchCall call;
            call.s = s;
            call.e = eU;
            call.hu = at(in + P, s4);
            if (!second) call.hu = mul2(call.hu, su);
            call.hv = at(in + 2 * P, s4);
            if (flip) call.hv = pr(-call.hv.x, -call.hv.y);
            call.su = su;
            call.j = r - 1;
            call.n = n;
            __syncwarp();
            march_row_general(S, call);
            s = call.s;
            R = call.R;
        }
        if (n >= 4) {
            float2 qe = o.sub(R.e, mul2(d2, R.fd0));
            float2 qu = o.add(R.hu, mul2(d2, R.r1)), qv = o.add(R.hv, mul2(d2, R.r2));
            if (second) {
                cp_async_wait_all();
                qe = mul2(c.half, o.add(at(QN, 0), qe));
                qu = mul2(c.half, o.add(at(QN, 256), qu));
                qv = mul2(c.half, o.add(at(QN, 512), qv));
            }
            if (__builtin_expect(p.r > 0.0f, 0)) {
                const float w = second ? 0.5f : 1.0f;
                const float2 hsum = o.add(R.e, R.Hm);
                const float C0 = 1.0f + w * march_friction(p, dt, hsum.x, R.hu.x, R.hv.x);
                const float C1 = 1.0f + w * march_friction(p, dt, hsum.y, R.hu.y, R.hv.y);
                qu = pr(qu.x / C0, qu.y / C1);
                qv = pr(qv.x / C0, qv.y / C1);
            }
            {
                // the final clamp (finish_cell) where a cell is not clearly wet
                const float2 hq = o.add(qe, R.Hm);
                if (__builtin_expect(any_lane(!(min_nan(hq.x, hq.y) > c.safe)), 0)) {
                    finish_cell(p, R.Hm.x, qe.x, qu.x, qv.x);
                    finish_cell(p, R.Hm.y, qe.y, qu.y, qv.y);
                }
            }
            if (second) {
                if (wide) {
                    if (o0) {   // an aligned pair of interior columns
                        *reinterpret_cast<float2*>(G.e_out + og) = qe;
                        *reinterpret_cast<float2*>(G.hu_out + og) = qu;
                        *reinterpret_cast<float2*>(G.hv_out + og) = qv;
                    }
                } else {
                    if (o0) { G.e_out[og] = qe.x; G.hu_out[og] = qu.x; G.hv_out[og] = qv.x; }
                    if (o1) { G.e_out[og + 1] = qe.y; G.hu_out[og + 1] = qu.y; G.hv_out[og + 1] = qv.y; }
                }
                if (__builtin_expect(x_images || (py && (r < 6 || r >= ny + 2)), 0)) {
                    if (o0) store_images(p, k, G, gx0, r - 2, qe.x, qu.x, qv.x);
                    if (o1) store_images(p, k, G, gx0 + 1, r - 2, qe.y, qu.y, qv.y);
                }
            } else {
                const unsigned t4 = march_stage(r - 2);
                at(ST, t4) = qe;
                at(ST + P, t4) = qu;
                at(ST + 2 * P, t4) = qv;
                if (__builtin_expect(wall_x, 0)) {
                    // ghost columns of Q* mirror the columns inside the wall
                    __syncwarp();
                    const int2 cq = S.col[0][lane];
                    float m[2][3];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const bool ghost = (i ? su.y : su.x) < 0.0f;
                        const int l = clampi((ghost ? (i ? cq.y : cq.x) : gx0 + i) - x0, 0, 63);
#pragma unroll
                        for (int q = 0; q < 3; ++q) m[i][q] = (&S.star[q][(r - 2) & (kMarchStage - 1)][0].x)[l];
                    }
                    __syncwarp();
                    at(ST, t4) = pr(m[0][0], m[1][0]);
                    at(ST + P, t4) = mul2(su, pr(m[0][1], m[1][1]));
                    at(ST + 2 * P, t4) = pr(m[0][2], m[1][2]);
                }
            }
        }
        if (__builtin_expect(south && !second && r == 5, 0)) idle = 3;
        ++r;
        march_barrier();
    }
    if (!second) cp_async_wait<0>();
}

}  // namespace goc

// Plain FP32 form over float4 "textures" with the reference's ghost layout: one kernel for Pass1 to Pass3, one for
// every level of both directions' cyclic reduction, one for the four boundary sides and one for GetStats.  This is
// the GPU restatement of timestep()/resetTimestep() (engine.cpp:849-1756) and of the compute.hlsl
// pixel shaders; it is compiled with -fmad=false so its arithmetic follows the FP32
// transcription operation by operation.  One domain per launch set.
#define CEL_EXACT_FP32 1
#include <cuda_runtime.h>

#include <mutex>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "boundary_plan.hpp"
#include "device_math.cuh"
#include "engine_iface.hpp"
#include "readback.hpp"
#include "scheme.hpp"

namespace cel {

namespace {

constexpr int BX2 = 32, BY2 = 8;

inline dim3 grid2(int w, int h) { return dim3((w + BX2 - 1) / BX2, (h + BY2 - 1) / BY2); }

// ---- Pass1 (compute.hlsl:380-458) at texel i: faces h,u,v {N,E,S,W} and the breaking slope ----
__device__ __forceinline__ void faces_of(const float4* __restrict__ st, const float4* __restrict__ bot, size_t i,
                                         const SimConsts& c, float4& h, float4& u, float4& v, float& msd) {
    const int NX = c.NX;
    const float4 cc = st[i], s = st[i - NX], n = st[i + NX], w = st[i - 1], e = st[i + 1];
    const float BN = bot[i].x, BE = bot[i].y, BS = bot[i - NX].x, BW = bot[i - 1].y;
    float wN, wE, wS, wW, huN, huE, huS, huW, hvN, hvE, hvS, hvW, sd;
    reconstruct_sd(c.two_theta, w.x, cc.x, e.x, wW, wE, sd);
    msd = sd * c.one_over_dx;
    reconstruct_sd(c.two_theta, s.x, cc.x, n.x, wS, wN, sd);
    msd = t_atan(fmaxf(msd, sd * c.one_over_dy));
    reconstruct(c.two_theta, w.y, cc.y, e.y, huW, huE);
    reconstruct(c.two_theta, s.y, cc.y, n.y, huS, huN);
    reconstruct(c.two_theta, w.z, cc.z, e.z, hvW, hvE);
    reconstruct(c.two_theta, s.z, cc.z, n.z, hvS, hvN);
    correct_w(BW, BE, cc.x, wW, wE);
    correct_w(BS, BN, cc.x, wS, wN);
    h = make_float4(wN - BN, wE - BE, wS - BS, wW - BW);
    float q;
    q = div_by_h(h.x, c.epsilon); u.x = q * huN; v.x = q * hvN;
    q = div_by_h(h.y, c.epsilon); u.y = q * huE; v.y = q * hvE;
    q = div_by_h(h.z, c.epsilon); u.z = q * huS; v.z = q * hvS;
    q = div_by_h(h.w, c.epsilon); u.w = q * huW; v.w = q * hvW;
}
// ... and its inundation / breaking record of a texel
__device__ __forceinline__ float4 aux_of(const float4& a1, const float4& h, float msd, const SimConsts& c) {
    const float mid = fmaxf((h.x + h.y + h.z + h.w) / 4.0f, a1.x);
    float bw = a1.w;
    if (msd > c.dissipation_threshold) bw = 1.0f;
    return make_float4(mid, 0.f, msd, bw);
}

// Pass1 into textures, region [1,nx+3)x[1,ny+3): only where the next pass must take the faces of a state
// that is about to change (addSolitaryWave does not rebuild them, engine.cpp:2154-2219).
__global__ void k_pass1(const float4* __restrict__ st, const float4* __restrict__ bot,
                        const float4* __restrict__ aux1, float4* __restrict__ H, float4* __restrict__ U,
                        float4* __restrict__ V, float4* __restrict__ aux2, SimConsts c) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int y = blockIdx.y * blockDim.y + threadIdx.y + 1;
    if (x >= c.nx + 3 || y >= c.ny + 3) return;
    const size_t i = size_t(y) * c.NX + x;
    float4 h, u, v;
    float msd;
    faces_of(st, bot, i, c, h, u, v, msd);
    H[i] = h; U[i] = u; V[i] = v;
    aux2[i] = aux_of(aux1[i], h, msd, c);
}

// ---- Pass2 (compute.hlsl:470-542): KP flux between the cell on a face's low side (m) and the one on
// its high side (p); x: the east face of m, y: its north face ----
__device__ __forceinline__ float3 x_flux(float hE, float uE, float vE, float hWe, float uWe, float vWe, float g, float hg) {
    const float cE = sqrtf(g * hE), cW = sqrtf(g * hWe);
    const float ap = fmaxf(fmaxf(uE + cE, uWe + cW), 0.f);
    const float am = fminf(fminf(uE - cE, uWe - cW), 0.f);
    return make_float3(numflux(ap, am, hWe * uWe, hE * uE, hWe - hE),
                       numflux(ap, am, hWe * (uWe * uWe + hg * hWe), hE * (uE * uE + hg * hE), hWe * uWe - hE * uE),
                       numflux(ap, am, hWe * uWe * vWe, hE * uE * vE, hWe * vWe - hE * vE));
}
__device__ __forceinline__ float3 y_flux(float hN, float uN, float vN, float hSn, float uSn, float vSn, float g, float hg) {
    const float cN = sqrtf(g * hN), cS = sqrtf(g * hSn);
    const float bp = fmaxf(fmaxf(vN + cN, vSn + cS), 0.f);
    const float bm = fminf(fminf(vN - cN, vSn - cS), 0.f);
    return make_float3(numflux(bp, bm, hSn * vSn, hN * vN, hSn - hN),
                       numflux(bp, bm, hSn * uSn * vSn, hN * uN * vN, hSn * uSn - hN * uN),
                       numflux(bp, bm, hSn * (vSn * vSn + hg * hSn), hN * (vN * vN + hg * hN), hSn * vSn - hN * vN));
}

struct Pass3Args {
    const float4* st; const float4* bot; const float4* H; const float4* U; const float4* V;
    const float4* aux2; float4* aux1;
    const float4* ABCx; const float4* ABCy;
    const float4* og; const float4* oog; const float2* ofg; const float2* oofg;   // F*, G* as pairs
    const float4* cur; const float4* pred; const float2* fgpred;
    float4* out; float4* sgrad; float2* sfg;
    float dt, dt_old, dt_old_old;
    float decay;   // pow(|white-water decay rate|, dt)
    int scheme;
};

// AdamsBashforthCoef (compute.hlsl:560-566)
__device__ __forceinline__ void ab_coef(float a, float b, float cc, float o[3]) {
    o[0] = (a / b) * ((2 * a + 6 * b + 3 * cc) / (b + cc)) + 6;
    o[1] = -(a / b) * ((2 * a + 3 * b + 3 * cc) / (cc));
    o[2] = (a / cc) * ((2 * a + 3 * b) / (b + cc));
}
// SecondOrderDerivatives (compute.hlsl:569-605)
__device__ __forceinline__ void second_order(float yn, float y1, float y2, float b, float cc, float o[3]) {
    float r = (2 * b + cc) / (b * (b + cc)), g = -(b + cc) / (b * cc), bb = (b) / (cc * (b + cc));
    o[0] = r * yn + g * y1 + bb * y2;
    r = (cc) / (b * (b + cc)); g = (b - cc) / (b * cc); bb = -(b) / (cc * (b + cc));
    o[1] = r * yn + g * y1 + bb * y2;
    r = -(cc) / (b * (b + cc)); g = (b + cc) / (b * cc); bb = -(b + 2 * cc) / (cc * (b + cc));
    o[2] = r * yn + g * y1 + bb * y2;
}

// ---- Pass1, Pass2 and Pass3Predictor (compute.hlsl:380-542, 616-812) in one kernel, every texel of the
// new state written once: zero on the ghost frame (engine.cpp:1007), the right-hand sides inside.  A CTA
// forms the faces of its 32 x 8 texels and the ring around them in shared memory, and a cell takes the
// fluxes of its four faces from there (each flux is computed by the two cells that share the face, from
// the same values), so neither the face nor the flux textures make a round trip through memory: 96 and 32
// bytes a cell and pass less, against 340 face computations for 256 cells.  STORED: the faces come from the
// textures (k_pass1).  The record's update runs on its own region [1,nx+2)x[1,ny+2).
// Bound by the IEEE divisions and square roots on small domains (latency) and by memory on large ones;
// event times: 512 x 64 cells Pass1, Pass2, Pass3 8.6 + 8.5 + 8.6 us and three clears -> 14.7 us, 1001 x 777
// 23 + 24 + 51 us and the clears -> 69 us. ----
constexpr int FW = BX2 + 2, FH = BY2 + 2;
template <bool STORED>
__global__ void __launch_bounds__(BX2 * BY2) k_pass123(Pass3Args a, SimConsts c) {
    __shared__ float4 fh[STORED ? 1 : FW * FH], fu[STORED ? 1 : FW * FH], fv[STORED ? 1 : FW * FH];
    __shared__ float fm[STORED ? 1 : FW * FH];
    const int x = blockIdx.x * BX2 + threadIdx.x;
    const int y = blockIdx.y * BY2 + threadIdx.y;
    const int NX = c.NX;
    const int f = (int(threadIdx.y) + 1) * FW + int(threadIdx.x) + 1;   // this cell in the tile
    if (!STORED) {
        const int xf = int(blockIdx.x * BX2) - 1, yf = int(blockIdx.y * BY2) - 1;
        for (int k = threadIdx.y * BX2 + threadIdx.x; k < FW * FH; k += BX2 * BY2) {
            const int gx = xf + k % FW, gy = yf + k / FW;
            if (gx < 1 || gy < 1 || gx >= c.nx + 3 || gy >= c.ny + 3) continue;
            faces_of(a.st, a.bot, size_t(gy) * NX + gx, c, fh[k], fu[k], fv[k], fm[k]);
        }
        __syncthreads();
    }
    if (x >= NX || y >= c.NY) return;
    const size_t i = size_t(y) * NX + x;
    if (x >= 1 && y >= 1 && x < c.nx + 2 && y < c.ny + 2) {
        const float4 a2 = STORED ? a.aux2[i] : aux_of(a.aux1[i], fh[f], fm[f], c);
        a.aux1[i] = make_float4(a2.x, 0.f, a2.z, a2.w * a.decay);
    }
    if (x < 2 || y < 2 || x >= c.nx + 2 || y >= c.ny + 2) {
        a.out[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    float3 xh, xw, yh, ys;
    {
        auto H = [&](int dx, int dy) { return STORED ? a.H[i + dx + ptrdiff_t(dy) * NX] : fh[f + dx + dy * FW]; };
        auto U = [&](int dx, int dy) { return STORED ? a.U[i + dx + ptrdiff_t(dy) * NX] : fu[f + dx + dy * FW]; };
        auto V = [&](int dx, int dy) { return STORED ? a.V[i + dx + ptrdiff_t(dy) * NX] : fv[f + dx + dy * FW]; };
        const float4 hc = H(0, 0), uc = U(0, 0), vc = V(0, 0);
        xh = x_flux(hc.y, uc.y, vc.y, H(1, 0).w, U(1, 0).w, V(1, 0).w, c.g, c.half_g);
        xw = x_flux(H(-1, 0).y, U(-1, 0).y, V(-1, 0).y, hc.w, uc.w, vc.w, c.g, c.half_g);
        yh = y_flux(hc.x, uc.x, vc.x, H(0, 1).z, U(0, 1).z, V(0, 1).z, c.g, c.half_g);
        ys = y_flux(H(0, -1).x, U(0, -1).x, V(0, -1).x, hc.z, uc.z, vc.z, c.g, c.half_g);
    }
    const float4* st = a.st;
    const float4* bot = a.bot;
    const float BYh = bot[i].x, BXh = bot[i].y, BAh = bot[i].z;
    const float BXw = bot[i - 1].y, BYs = bot[i - NX].x;
    const float4 cc = st[i], r = st[i + 1], l = st[i - 1], u = st[i + NX], d = st[i - NX];
    const float4 cx = a.ABCx[i], cy = a.ABCy[i];
    const float sl = c.sea_level;
    const float h = fmaxf(0.f, cc.x - BAh);
    const float dh = fmaxf(0.f, sl - BAh), d2 = dh * dh, d3 = d2 * dh;
    const float dl = fmaxf(0.f, sl - bot[i - 1].z), dr = fmaxf(0.f, sl - bot[i + 1].z);
    const float ddn = fmaxf(0.f, sl - bot[i - NX].z), du = fmaxf(0.f, sl - bot[i + NX].z);
    const float dll = fmaxf(0.f, sl - bot[i - 2].z), drr = fmaxf(0.f, sl - bot[i + 2].z);
    const float ddd = fmaxf(0.f, sl - bot[i - 2 * NX].z), duu = fmaxf(0.f, sl - bot[i + 2 * NX].z);
    const float e0 = cc.x - sl;
    const float el = l.x - sl, er = r.x - sl, ed = d.x - sl, eu = u.x - sl;
    const float ell = st[i - 2].x - sl, err = st[i + 2].x - sl;
    const float edd = st[i - 2 * NX].x - sl, euu = st[i + 2 * NX].x - sl;
    const float eul = st[i + NX - 1].x - sl, eur = st[i + NX + 1].x - sl;
    const float edl = st[i - NX - 1].x - sl, edr = st[i - NX + 1].x - sl;
    const float odx = c.one_over_dx, ody = c.one_over_dy;
    const float od2x = odx * odx, od3x = od2x * odx, od2y = ody * ody, od3y = od2y * ody;
    const float ddx = (-drr + 8 * dr - 8 * dl + dll) * odx / 12.0f;
    const float ddy = (-duu + 8 * du - 8 * ddn + ddd) * ody / 12.0f;
    const float exy = (0.25f * odx * ody * (eur - edr - eul + edl));
    const float exx = od2x * (er - 2 * e0 + el);
    const float eyy = od2y * (eu - 2 * e0 + ed);
    const float Bg = c.Bcoef_g;
    const float P1x = Bg * (d3) * ((err - 2 * er + 2 * el - ell) * (0.5f * od3x) +
                                   (eur - eul - 2 * er + 2 * el + edr - edl) * (0.5f * odx * od2y));
    const float P2x = Bg * (d2) * (ddx * (2 * exx + eyy) + ddy * exy);
    const float P1y = Bg * (d3) * ((euu - 2 * eu + 2 * ed - edd) * (0.5f * od3y) +
                                   (eur + eul - 2 * eu + 2 * ed - edr - edl) * (0.5f * ody * od2x));
    const float P2y = Bg * (d2) * (ddy * (exx + 2 * eyy) + ddx * exy);
    // Both friction laws give 0 * |momentum| for a zero coefficient, whatever the (finite) depth: the two
    // double-precision powers are left out then (h - h carries a depth that is not finite).
    const float fr = c.friction == 0.f ? 0.f * sqrtf(cc.y * cc.y + cc.z * cc.z) + (h - h)
                                       : friction_calc(cc.y, cc.z, h, c.friction, c.is_manning, c.g, c.epsilon);
    const float s1 = -c.g_over_dx * h * (BXh - BXw) - cc.y * fr + (P1x + P2x);
    const float s2 = -c.g_over_dy * h * (BYh - BYs) - cc.z * fr + (P1y + P2y);
    const float f0 = (xw.x - xh.x) * odx + (ys.x - yh.x) * ody + 0.f;
    const float f1 = (xw.y - xh.y) * odx + (ys.y - yh.y) * ody + s1;
    const float f2 = (xw.z - xh.z) * odx + (ys.z - yh.z) * ody + s2;
    const float sixth = 1.0f / 6.0f;
    const float Fs = (sixth * dh * (ddx * ((ody / 2.0f) * (u.z - d.z)) + (ddy * ((odx / 2.0f) * (r.z - l.z)))));
    const float Gs = (sixth * dh * (ddx * ((ody / 2.0f) * (u.y - d.y)) + (ddy * ((odx / 2.0f) * (r.y - l.y)))));
    const float dt = a.dt;
    float wO = 0.f, huO = 0.f, hvO = 0.f;
    if (a.scheme == CEL_SCHEME_EULER) {
        wO = cc.x + dt * f0;
        huO = cx.x * l.y + cx.y * cc.y + cx.z * r.y + dt * f1;
        hvO = cy.x * d.z + cy.y * cc.z + cy.z * u.z + dt * f2;
    } else {
        const float4 o = a.og[i], oo = a.oog[i];
        const float2 fo = a.ofg[i], foo = a.oofg[i];
        if (a.scheme == CEL_SCHEME_PREDICTOR) {
            wO = cc.x + dt / 12.0f * (23.0f * f0 - 16.0f * o.x + 5.0f * oo.x);
            huO = cx.x * l.y + cx.y * cc.y + cx.z * r.y + dt / 12.0f * (23.0f * f1 - 16.0f * o.y + 5.0f * oo.y) +
                  (2.0f * Fs - 3.0f * fo.x + foo.x);
            hvO = cy.x * d.z + cy.y * cc.z + cy.z * u.z + dt / 12.0f * (23.0f * f2 - 16.0f * o.z + 5.0f * oo.z) +
                  (2.0f * Gs - 3.0f * fo.y + foo.y);
        } else if (a.scheme == CEL_SCHEME_PREDICTOR_ADAPTIVE) {
            float cf[3], dF[3], dG[3];
            ab_coef(dt, a.dt_old, a.dt_old_old, cf);
            second_order(Fs, fo.x, foo.x, a.dt_old, a.dt_old_old, dF);
            second_order(Gs, fo.y, foo.y, a.dt_old, a.dt_old_old, dG);
            wO = cc.x + dt / 6.0f * (cf[0] * f0 + cf[1] * o.x + cf[2] * oo.x);
            huO = cx.x * l.y + cx.y * cc.y + cx.z * r.y + dt / 6.0f * (cf[0] * f1 + cf[1] * o.y + cf[2] * oo.y) +
                  dt / 6.0f * (cf[0] * dF[0] + cf[1] * dF[1] + cf[2] * dF[2]);
            hvO = cy.x * d.z + cy.y * cc.z + cy.z * u.z + dt / 6.0f * (cf[0] * f2 + cf[1] * o.z + cf[2] * oo.z) +
                  dt / 6.0f * (cf[0] * dG[0] + cf[1] * dG[1] + cf[2] * dG[2]);
        } else {  // corrector
            const float4 qc = a.cur[i], qr = a.cur[i + 1], ql = a.cur[i - 1], qu = a.cur[i + NX], qd = a.cur[i - NX];
            const float4 pr = a.pred[i];
            const float2 fp = a.fgpred[i];
            wO = qc.x + dt / 24.0f * (9 * f0 + 19 * pr.x - 5 * o.x + 1 * oo.x);
            huO = cx.x * ql.y + cx.y * qc.y + cx.z * qr.y + dt / 24.0f * (9 * f1 + 19 * pr.y - 5 * o.y + 1 * oo.y) + Fs -
                  fp.x;
            hvO = cy.x * qd.z + cy.y * qc.z + cy.z * qu.z + dt / 24.0f * (9 * f2 + 19 * pr.z - 5 * o.z + 1 * oo.z) + Gs -
                  fp.y;
        }
    }
    a.out[i] = make_float4(wO, huO, hvO, 0.f);
    a.sgrad[i] = make_float4(f0, f1, f2, 0.f);
    a.sfg[i] = make_float2(Fs, Gs);
}

// ---- Cyclic reduction (compute.hlsl:835-947), every level of a system in one CTA -----------
// The levels of one direction, level k's elements i = 0 .. len_k - 1 (texel i + 2):
//   reduce      D_k[i] = D_{k-1}[2i+1] - D_{k-1}[2i] k1 - D_{k-1}[2i+2] k2
//   substitute  X_k[2j] = (D_k[2j] - a X_{k+1}[j-1] - c X_{k+1}[j]) / b,  X_k[2j+1] = X_{k+1}[j]
// with zeros where an index leaves the level.  k1 and k2 are the shader's quotients of coefficient
// texels: they depend on the bottom only, so the host forms them once (the same IEEE divisions); the
// division by b stays a division.  Operation by operation this is the shader's arithmetic, so the
// results do not change a bit.
//
// A draw per level, the shader's way, costs 2 log2(n) launches a direction, most of which touch a
// few elements.  Here a CTA keeps a system's levels in shared memory: the first CTAs take CR_COLS
// adjacent columns each (whose level 0 they read from the state when they need it instead of keeping it),
// the others one row.  What bounds it is latency, since the levels are a serial chain: the coefficients of
// a level are loaded before the barrier that ends the level before it, and levels of at most 32
// elements run in one warp.  hu and hv go back into the state in place (CopyFromXxAndXy,
// compute.hlsl:814-823, is folded in).  Measured by event timing, a pass's solves: 512 x 64 cells 32
// launches and 210 us -> 14.7 us, 1001 x 777 cells 38 launches and 295 us -> 42 us.
constexpr int CR_MAX_LEVELS = 16;
constexpr int CR_THREADS = 256;
constexpr int CR_COLS = 4;              // columns of a column CTA: 64-byte pieces of a state row
constexpr size_t CR_SMEM_MAX = 200 * 1024;
constexpr int CR_TALL_THREADS = 1024;
constexpr int CR_TALL_COLS = 296, CR_TALL_ROWS = 4096;   // domains whose columns k_cr_tall takes
struct CrLevels {
    int K;                              // levels
    int tail;                           // first level (>= 1) that one warp handles
    int len[CR_MAX_LEVELS];
    int off[CR_MAX_LEVELS];             // start of a level's values in a system's scratch
    size_t koff[CR_MAX_LEVELS];         // start of a level's {k1, k2} (levels >= 1)
    size_t soff[CR_MAX_LEVELS];         // start of a level's {a, c, b}, even elements only
    int total;                          // scratch values of a system
    const float2* k12;                  // rows: [y][i], columns: [i][x]
    const float4* acb;
};
struct SolveArgs {
    float4* st;
    CrLevels x, y;
    int bands;                          // column CTAs of k_cr
    float* scratch;                     // the levels in global memory where shared memory does not hold them
};

// ROW: one row (level 0 kept with the levels, W = 1); else W columns.  lv: the levels, element i of
// column c of level k at lv[(off_k + i) * W + c]; st0: the level-0 values in the state, d0 floats apart;
// sys: the row, or this thread's column; ns: the number of columns (the columns' coefficient stride).
template <bool ROW, int W, int THREADS>
__device__ __forceinline__ void cr_solve(const CrLevels& L, float* __restrict__ lv, float* st0, size_t d0, int sys, int ns,
                                         bool live) {
    constexpr int T = THREADS / W;
    const int c = int(threadIdx.x) % W, t = int(threadIdx.x) / W;
    const int n = L.len[0];
    lv += c;
    auto k12 = [&](int k, int i) -> float2 {
        if (!live || i >= L.len[k]) return make_float2(0.f, 0.f);
        return __ldg(L.k12 + L.koff[k] + (ROW ? size_t(sys) * L.len[k] + i : size_t(i) * ns + sys));
    };
    auto acb = [&](int k, int j) -> float4 {
        const int half = (L.len[k] + 1) / 2;
        if (!live || j >= half) return make_float4(0.f, 0.f, 1.f, 0.f);
        return __ldg(L.acb + L.soff[k] + (ROW ? size_t(sys) * half + j : size_t(j) * ns + sys));
    };
    auto d0_at = [&](int i) -> float {
        if (ROW) return lv[L.off[0] + i];
        return (live && i < n) ? st0[size_t(i) * d0] : 0.f;
    };
    auto reduce = [&](int k, int i, float2 q) {
        const float* p = lv + size_t(L.off[k - 1]) * W;
        const float mid = k == 1 ? d0_at(2 * i + 1) : p[(2 * i + 1) * W];
        const float lo = k == 1 ? d0_at(2 * i) : p[(2 * i) * W];
        const float hi = k == 1 ? d0_at(2 * i + 2) : p[(2 * i + 2) * W];
        lv[size_t(L.off[k] + i) * W] = mid - lo * q.x - hi * q.y;
    };
    auto substitute = [&](int k, int j, float4 q) {
        const bool last = k + 1 == L.K;
        const float* xn = last ? nullptr : lv + size_t(L.off[k + 1]) * W;
        const float x1 = (!last && j > 0) ? xn[(j - 1) * W] : 0.f;
        const float x2 = (!last && j < L.len[k + 1]) ? xn[j * W] : 0.f;
        const float d = k == 0 ? d0_at(2 * j) : lv[size_t(L.off[k] + 2 * j) * W];
        const float o = (d - q.x * x1 - q.y * x2) / q.z;
        if (k == 0) {
            if (live) {
                st0[size_t(2 * j) * d0] = o;
                if (2 * j + 1 < n) st0[size_t(2 * j + 1) * d0] = x2;
            }
        } else {
            lv[size_t(L.off[k] + 2 * j) * W] = o;
            if (2 * j + 1 < L.len[k]) lv[size_t(L.off[k] + 2 * j + 1) * W] = x2;
        }
    };
    float2 q = L.K > 1 ? k12(1, t) : make_float2(0.f, 0.f);
    if (ROW) {
        for (int i = t; i < n; i += T) lv[L.off[0] + i] = st0[size_t(i) * d0];
        if (t == 0) lv[L.off[0] + n] = 0.f;
        __syncthreads();
    }
    for (int k = 1; k < L.tail; ++k) {
#pragma unroll 4
        for (int i = t; i < L.len[k]; i += T) reduce(k, i, i == t ? q : k12(k, i));
        if (t == 0) lv[size_t(L.off[k] + L.len[k]) * W] = 0.f;
        if (k + 1 < L.K) q = k12(k + 1, t);
        __syncthreads();
    }
    float4 s = make_float4(0.f, 0.f, 1.f, 0.f);
    if (threadIdx.x < 32) {   // levels of at most 32 elements, all columns together
        for (int k = L.tail; k < L.K; ++k) {
            if (t < L.len[k]) reduce(k, t, q);
            if (t == 0) lv[size_t(L.off[k] + L.len[k]) * W] = 0.f;
            if (k + 1 < L.K) q = k12(k + 1, t);
            __syncwarp();
        }
        for (int k = L.K - 1; k >= L.tail; --k) {
            s = acb(k, t);
            if (2 * t < L.len[k]) substitute(k, t, s);
            __syncwarp();
        }
    }
    s = acb(L.tail - 1, t);
    __syncthreads();
    for (int k = L.tail - 1; k >= 0; --k) {
#pragma unroll 4
        for (int j = t; 2 * j < L.len[k]; j += T) substitute(k, j, j == t ? s : acb(k, j));
        if (k > 0) {
            s = acb(k - 1, t);
            __syncthreads();
        }
    }
}

// A level's coefficients as k_cr reads them, from its textures (2 texels of border; pitch len + 4 in rows, NX in
// columns): for equation i of system s the two multipliers, from the level before, and for every second
// one its own three.
__global__ void k_pack_level(const float4* __restrict__ prev, const float4* __restrict__ cur, bool rows, int n, int len,
                             int prev_pitch, int NX, float2* __restrict__ k12, float4* __restrict__ acb) {
    const size_t e = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e >= size_t(len) * n) return;
    const int s = int(rows ? e / len : e % n), i = int(rows ? e % len : e / n);
    if (prev) {
        const size_t si = rows ? 1 : NX;
        const float4* p = prev + size_t(s + 2) * (rows ? prev_pitch : 1) + size_t(2 * i + 2) * si;
        k12[e] = make_float2(p[si].x / p[0].y, p[si].z / p[2 * si].y);
    }
    const int half = (len + 1) / 2;
    if (i < half) {
        const float4 q = cur[size_t(s + 2) * (rows ? len + 4 : 1) + size_t(2 * i + 2) * (rows ? 1 : NX)];
        acb[rows ? size_t(s) * half + i : size_t(i) * n + s] = make_float4(q.x, q.z, q.y, 0.f);
    }
}

// SMEM_X / SMEM_Y: the rows' / the columns' levels fit in shared memory.
template <bool SMEM_X, bool SMEM_Y>
__global__ void __launch_bounds__(CR_THREADS) k_cr(SolveArgs a, SimConsts c) {
    extern __shared__ float cr_sm[];
    // columns first: a column CTA has four systems and the strided reads
    const int rows = c.ny, bands = a.bands, b = int(blockIdx.x) - bands;
    if (b >= 0) {
        float* lv = SMEM_X ? cr_sm : a.scratch + size_t(b) * a.x.total;
        cr_solve<true, 1, CR_THREADS>(a.x, lv, reinterpret_cast<float*>(a.st + size_t(b + 2) * c.NX + 2) + 1, 4, b, 0, true);
    } else {
        const int band = blockIdx.x, col = band * CR_COLS + int(threadIdx.x) % CR_COLS;
        float* lv = SMEM_Y ? cr_sm
                           : a.scratch + (SMEM_X ? 0 : size_t(rows) * a.x.total) + size_t(band) * a.y.total * CR_COLS;
        cr_solve<false, CR_COLS, CR_THREADS>(a.y, lv, reinterpret_cast<float*>(a.st + size_t(2) * c.NX + 2 + col) + 2, size_t(4) * c.NX, col, c.nx,
                        col < c.nx);
    }
}

// Few tall columns: a CTA of 1024 threads per column, in a launch of its own before the rows'.  What bounds
// tall columns is the serial sweep of a level by the 64 threads that a column has in k_cr, and beside it the
// rows' CTAs, one or two an SM, since a launch's CTAs all take the shared memory that four columns' levels
// need.  Level 0 comes 4 bytes a 32-byte sector, so columns that fill the GPU are better off in fours.
// Event times of the solves, k_cr -> both launches: 8 x 4096 cells 69 -> 45 us, 64 x 8192 509 -> 141, 148 x
// 12000 937 -> 244, 8 x 32768 636 -> 269, 296 x 4096 154 -> 130; below 4096 rows it is the other way: 64 x 1000
// 31 -> 35.  (A launch per level and direction took longer than k_cr except on such columns: 2 x 32768 cells
// 697 us a step, 1391 in k_cr, 569 here.)
__global__ void __launch_bounds__(CR_TALL_THREADS) k_cr_tall(SolveArgs a, SimConsts c) {
    extern __shared__ float cr_sm[];
    const int col = blockIdx.x;
    cr_solve<false, 1, CR_TALL_THREADS>(a.y, cr_sm, reinterpret_cast<float*>(a.st + size_t(2) * c.NX + 2 + col) + 2,
                                        size_t(4) * c.NX, col, c.nx, true);
}

// ---- Boundaries (compute.hlsl:985-1309) --------------------------------------------------
struct BArgs {
    int side;  // 0 = N, 1 = E, 2 = S, 3 = W
    int type, width;
    float sea_level, amp, period, theta;
    float uts_eta, uts_hu, uts_hv;
    int n_waves, nleaf;
    const float4* waves;
    float t, dt;
    int x0, y0, sw, sh;
};

// Pairwise tree sum of the irregular-wave components over 2^(K-1) leaves
// (ColumnSumReduce / RowSumReduce, compute.hlsl:1196-1212): a binary-counter stack gives the
// balanced-tree association; runs of constant components (sea level, 0, 0) are pushed as whole
// aligned subtrees.
__device__ float3 irregular_sum(const BArgs& b, float xx, float yy, float dh, float g) {
    float3 stk[17];
    int sz[17];
    int top = 0;
    const bool wet = dh > CEL_MIN_DEPTH;
    const int nreal = wet ? min(b.n_waves, b.nleaf) : 0;
    int m = 0;
    while (m < b.nleaf) {
        float3 v;
        int s;
        if (m < nreal) {
            float e, hu, hv;
            const float4 wv = b.waves[m];
            sine_wave(xx, yy, b.t, dh, wv.x, wv.y, wv.z, wv.w, g, e, hu, hv);
            v = make_float3(e + b.sea_level, hu, hv);
            s = 1;
        } else {
            s = (m == 0) ? b.nleaf : (m & -m);
            while (m + s > b.nleaf) s >>= 1;
            v = make_float3(float(s) * b.sea_level, 0.f, 0.f);
        }
        m += s;
        stk[top] = v;
        sz[top] = s;
        ++top;
        while (top >= 2 && sz[top - 1] == sz[top - 2]) {
            const float3 r = stk[top - 1], l = stk[top - 2];
            stk[top - 2] = make_float3(l.x + r.x, l.y + r.y, l.z + r.z);
            sz[top - 2] *= 2;
            --top;
        }
    }
    return stk[0];
}

// The value one side's shader writes at texel (x, y)
__device__ float4 boundary_value(const float4* st, const float4* __restrict__ bot, const BArgs& b, const SimConsts& c, int x,
                                 int y) {
    const int NX = c.NX, NY = c.NY;
    const size_t i = size_t(y) * NX + x;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    const float sl = b.sea_level;
    if (b.type == CEL_BC_SOLID) {
        int qx, qy;
        solid_source(b.side, x, y, c.nx, c.ny, qx, qy);
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);  // out-of-range texture loads read zero
        if (qx >= 0 && qy >= 0 && qx < NX && qy < NY) s = st[size_t(qy) * NX + qx];
        o.x = s.x;
        o.y = (b.side == 1 || b.side == 3) ? -s.y : s.y;
        o.z = (b.side == 0 || b.side == 2) ? -s.z : s.z;
    } else if (b.type == CEL_BC_SPONGE) {
        const float dh = fmaxf(CEL_MIN_DEPTH, sl - bot[i].z);
        float L, dist;
        if (b.side == 3) { L = float(b.width) * c.dx; dist = float(x) * c.dx; }
        else if (b.side == 1) { L = float(b.width) * c.dx; dist = float(NX - x) * c.dx; }
        else if (b.side == 2) { L = float(b.width) * c.dy; dist = float(y) * c.dy; }
        else { L = float(b.width) * c.dy; dist = float(NY - y) * c.dy; }
        const float gam = sponge_fn(L, dist) / sponge_fn(L, dist + sqrtf(c.g * dh) * b.dt);
        const float4 s = st[i];
        o.x = gam * (s.x - sl) + sl;
        o.y = gam * s.y;
        o.z = gam * s.z;
    } else if (b.type == CEL_BC_SINEWAVE) {
        const float dh = fmaxf(0.f, sl - bot[i].z);
        const float xx = (b.side == 1) ? float(x - NX) * c.dx : float(x) * c.dx;
        const float yy = (b.side == 0) ? float(y - NY) * c.dy : float(y) * c.dy;
        float e = 0.f, hu = 0.f, hv = 0.f;
        if (dh > CEL_MIN_DEPTH) sine_wave(xx, yy, b.t, dh, b.amp, b.period, b.theta, 0.f, c.g, e, hu, hv);
        o.x = e + sl; o.y = hu; o.z = hv;
    } else if (b.type == CEL_BC_UTS) {
        o.x = b.uts_eta + sl; o.y = b.uts_hu; o.z = b.uts_hv;
    } else {  // irregular waves: one component per texel along the side, tree-summed
        const bool colwise = (b.side == 1 || b.side == 3);
        const int along = colwise ? y : x;
        const int lim = colwise ? c.ny : c.nx;
        if (along >= 2 && along < lim + 2) {
            const float dh = fmaxf(0.f, sl - bot[i].z);
            const float xx = (b.side == 1) ? float(x - NX) * c.dx : float(x) * c.dx;
            const float yy = (b.side == 0) ? float(y - NY) * c.dy : float(y) * c.dy;
            const float3 r = irregular_sum(b, xx, yy, dh, c.g);
            o.x = r.x; o.y = r.y; o.z = r.z;
        }
    }
    return o;
}

__global__ void k_boundary(const float4* __restrict__ st, const float4* __restrict__ bot, float4* __restrict__ strip,
                           BArgs b, SimConsts c) {
    const int sx = blockIdx.x * blockDim.x + threadIdx.x;
    const int sy = blockIdx.y * blockDim.y + threadIdx.y;
    if (sx >= b.sw || sy >= b.sh) return;
    strip[size_t(sy) * b.sw + sx] = boundary_value(st, bot, b, c, b.x0 + sx, b.y0 + sy);
}

__global__ void k_strip_copy(float4* __restrict__ st, const float4* __restrict__ strip, int x0, int y0, int sw, int sh,
                             int NX) {
    const int sx = blockIdx.x * blockDim.x + threadIdx.x;
    const int sy = blockIdx.y * blockDim.y + threadIdx.y;
    if (sx >= sw || sy >= sh) return;
    st[size_t(y0 + sy) * NX + x0 + sx] = strip[size_t(sy) * sw + sx];
}

// All four sides in one launch (boundary_plan.hpp): a work item is 256 texels of a segment, written in
// place by one thread each, or a whole corner, whose two sides one CTA takes in drawing order.  The
// sides' own launches, each followed by a copy out of the strip texture, are 8 launches of a few
// hundred texels each; domains that the plan refuses still take them.
struct BoundaryArgs {
    BArgs side[4];
    Rect region[BND_REGIONS];
};
__global__ void __launch_bounds__(256) k_boundary_all(float4* st, const float4* __restrict__ bot, const int2* __restrict__ items,
                                                      BoundaryArgs a, SimConsts c) {
    const int2 it = items[blockIdx.x];
    const Rect r = a.region[it.x];
    if (it.x < 4) {
        const int w = r.x1 - r.x0, k = it.y + int(threadIdx.x);
        if (k >= w * (r.y1 - r.y0)) return;
        const int x = r.x0 + k % w, y = r.y0 + k / w;
        st[size_t(y) * c.NX + x] = boundary_value(st, bot, a.side[it.x], c, x, y);
        return;
    }
    for (int q = 0; q < 2; ++q) {
        const BArgs& b = a.side[corner_side(it.x - 4, q)];
        const int x0 = max(r.x0, b.x0), x1 = min(r.x1, b.x0 + b.sw), y0 = max(r.y0, b.y0), y1 = min(r.y1, b.y0 + b.sh);
        const int w = x1 - x0, n = w > 0 ? w * (y1 - y0) : 0;
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
            const int x = x0 + k % w, y = y0 + k / w;
            st[size_t(y) * c.NX + x] = boundary_value(st, bot, b, c, x, y);
        }
        __syncthreads();
    }
}

// ---- GetStats (compute.hlsl:1319-1378) and its FP64 reduction in one launch -------------
// A lane per cell, 16 lanes per 4x4 block: every lane forms its cell's terms, and the block's sums
// take them in the shader's order from the lanes (the texture's partial sums, kept for getWaterHeight, do
// not change a bit).  Blocks cut off by the far edges count for the FP64 volume and the non-finite flag
// only.  Each CTA leaves one set of FP64 partials, and the last one to finish adds them up in CTA order, so
// the totals do not depend on scheduling.  A thread per block chained 16 cells' divisions and roots (16.9 us
// by event timing on 512 x 64 cells), and the reduction by one CTA over every cell before that took 313 us
// on 1001 x 777.
// out: [0..4] sums, [5..8] maxima, [9] the volume, [10] 1 if a state value is not finite
constexpr int STATS_THREADS = 256;
constexpr int STATS_CTAS = 592;   // at most: 4 per SM
__global__ void __launch_bounds__(STATS_THREADS) k_stats(const float4* __restrict__ st, const float4* __restrict__ bot,
                                                         float* __restrict__ blocks, SimConsts c, double* __restrict__ part,
                                                         unsigned int* __restrict__ done, double* __restrict__ out) {
    __shared__ double sm[STATS_THREADS / 32][11];
    __shared__ bool last;
    const int nbx = c.nx / 4, nby = c.ny / 4, tbx = (c.nx + 3) / 4, tby = (c.ny + 3) / 4;
    const int lane = threadIdx.x & 31, cell = lane & 15;
    double v[11] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    // (the trip count is the same for a CTA: the shuffles need whole warps)
    for (int k0 = blockIdx.x * (STATS_THREADS / 16); k0 < tbx * tby; k0 += gridDim.x * (STATS_THREADS / 16)) {
        const int k = k0 + int(threadIdx.x >> 4);   // block
        const int bx = k % tbx, by = k / tbx, x = 4 * bx + (cell & 3), y = 4 * by + (cell >> 2);
        const bool here = by < tby && x < c.nx && y < c.ny, whole = bx < nbx && by < nby;
        float q[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (here) {
            const size_t i = size_t(y + 2) * c.NX + x + 2;
            const float4 s = st[i];
            const float B = bot[i].z;
            if (!isfinite(s.x) || !isfinite(s.y) || !isfinite(s.z)) v[10] = 1.0;
            v[9] += fmax(0.0, double(s.x) - double(B));
            const float h = fmaxf(0.f, s.x - B);
            const float cc = sqrtf(c.g * h);
            const float d = div_by_h(h, c.epsilon);
            const float u = d * s.y, w = d * s.z;
            const float u2v2 = u * u + w * w;
            q[0] = h; q[1] = h * (B + 0.5f * h); q[2] = s.y; q[3] = s.z;
            q[4] = (s.y * u + s.z * w);
            q[5] = u2v2; q[6] = h;
            q[7] = fmaxf((fabsf(u) + cc) * c.one_over_dx, (fabsf(w) + cc) * c.one_over_dy);
            q[8] = u2v2 * d;
        }
        float sum[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int t = 0; t < 16; ++t)
            for (int m = 0; m < 5; ++m) sum[m] += __shfl_sync(0xffffffffu, q[m], (lane & 16) + t);
        for (int off = 8; off; off >>= 1)
            for (int m = 5; m < 9; ++m) q[m] = fmaxf(q[m], __shfl_xor_sync(0xffffffffu, q[m], off));
        if (whole && cell == 0) {
            float* o = blocks + (size_t(by) * nbx + bx) * 9;
            for (int m = 0; m < 5; ++m) { o[m] = sum[m]; v[m] += double(sum[m]); }
            for (int m = 5; m < 9; ++m) { o[m] = fmaxf(0.f, q[m]); v[m] = fmax(v[m], double(o[m])); }
        }
    }
    auto is_max = [](int m) { return (m >= 5 && m < 9) || m == 10; };
    auto cta_reduce = [&]() {   // thread 0 ends with the CTA's totals
        for (int m = 0; m < 11; ++m) {
            double a = v[m];
            for (int off = 16; off; off >>= 1) {
                const double o = __shfl_down_sync(0xffffffffu, a, off);
                a = is_max(m) ? fmax(a, o) : a + o;
            }
            if (lane == 0) sm[threadIdx.x >> 5][m] = a;
        }
        __syncthreads();
        if (threadIdx.x < 11) {
            const int m = threadIdx.x;
            double a = sm[0][m];
            for (int w = 1; w < STATS_THREADS / 32; ++w) a = is_max(m) ? fmax(a, sm[w][m]) : a + sm[w][m];
            v[0] = a;   // thread m holds total m
        }
    };
    cta_reduce();
    if (threadIdx.x < 11) {
        part[size_t(blockIdx.x) * 11 + threadIdx.x] = v[0];
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int m = 0; m < 11; ++m) v[m] = 0.0;
    for (int b = threadIdx.x; b < int(gridDim.x); b += STATS_THREADS)
        for (int m = 0; m < 11; ++m) {
            const double a = __ldcg(part + size_t(b) * 11 + m);
            v[m] = is_max(m) ? fmax(v[m], a) : v[m] + a;
        }
    __syncthreads();   // the first reduction's reads of sm are done
    cta_reduce();
    if (threadIdx.x < 11) out[threadIdx.x] = v[0];
    if (threadIdx.x == 0) *done = 0u;
}

// AddSolitaryWave (compute.hlsl:949-976) over [1,nx+3)x[1,ny+3), reading a copy of the state
__global__ void k_add_solitary(const float4* __restrict__ copy, const float4* __restrict__ bot, float4* __restrict__ st,
                               SimConsts c, float H, float th, float xc, float yc) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int y = blockIdx.y * blockDim.y + threadIdx.y + 1;
    if (x >= c.nx + 3 || y >= c.ny + 3) return;
    const size_t i = size_t(y) * c.NX + x;
    const float4 s = copy[i];
    const float depth = fmaxf(s.x - bot[i].z, 0.f);
    const float K = sqrtf(0.75f * fabsf(H) / t_pow(depth, 3.0f));
    const float C = sqrtf(c.g * (H + depth));
    const float ch = t_cosh(K * ((float(x) * c.dx - xc) * t_cos(th) + (float(y) * c.dy - yc) * t_sin(th)));
    const float e = H * 1.0f / t_pow(ch, 2.0f);
    st[i] = make_float4(s.x + e, s.y + C * t_cos(th) * e, s.z + C * t_sin(th) * e, 0.f);
}

// ---------------------------------------------------------------------------------------------
class PlainEngine : public EngineIface {
public:
    cel_params p{};
    HostSetup hs;
    SimConsts c{};
    Scheme sch;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    cudaStream_t sstream = nullptr;          // the statistics run beside the pass that they precede
    cudaEvent_t ev_state = nullptr, ev_stats = nullptr;
    bool stats_pending = false;              // ... and the engine's stream has not waited for them yet
    KernelTimer tm;
    Readback rb;
    size_t ntex = 0;
    // device textures
    // The state rotates through three textures and the derivatives through four, by index: a corrector
    // finds the state that it corrects and the predictor's derivatives where their passes left them
    // (the reference copies them aside, engine.cpp:1050-1058: 48 bytes a cell and predictor).
    float4 *st[3] = {nullptr, nullptr, nullptr}, *H = nullptr, *U = nullptr, *V = nullptr;
    float4 *AUX1 = nullptr, *AUX2 = nullptr, *BOT = nullptr;
    float4 *GRAD[4] = {nullptr, nullptr, nullptr, nullptr}, *STRIP = nullptr;
    float2* FG[4] = {nullptr, nullptr, nullptr, nullptr};
    float4* WAVES = nullptr;
    float4 *ABCx = nullptr, *ABCy = nullptr;                        // level-0 systems (the right-hand sides' products)
    float2 *K12x = nullptr, *K12y = nullptr;                        // reduction multipliers of every level
    float4 *ACBx = nullptr, *ACBy = nullptr;                        // substitution coefficients of every level
    SolveArgs solve{};
    bool smem_x = true, smem_y = true;
    size_t smem_cr = 0, smem_tall = 0;
    bool tall = false;                                              // k_cr_tall takes the columns
    bool planned = false;                                           // the four sides run as one launch
    Rect regions[BND_REGIONS] = {};
    int2* bitems = nullptr;
    int nbitems = 0;
    float* blocks = nullptr;
    double* dstats = nullptr;
    double* spart = nullptr;
    unsigned int* sdone = nullptr;
    int stats_ctas = 1;
    std::vector<void*> allocs;
    int wave_off[4] = {0, 0, 0, 0};
    int sim_idx = 0, cur_i = 0, old_i = 0, oldold_i = 1, scratch_i = 2, spare_i = 3, pred_i = 3;
    int uts_iter[4] = {1, 1, 1, 1};
    // Faces belong to the current state (the pass forms them) unless a solitary wave was added since the last
    // pass: the reference built them at the end of that pass and does not rebuild them then.
    bool faces_pending = false;   // a pass has run since the last remesh, state or terrain change
    bool faces_stored = false;    // H, U, V and AUX2 hold the faces of the state before the wave
    std::vector<float> terrain;   // bathymetry grid given by set_bathymetry (used by remesh)
    int terrain_nx = 0, terrain_ny = 0;
    // stats bookkeeping for the latest device-side GetStats
    int last_stats_scheme = 0;
    float last_stats_dt = 0, last_stats_time = 0;

    ~PlainEngine() override {
        for (void* a : allocs) cudaFree(a);
        for (cel_boundary* b : {&p.west, &p.east, &p.south, &p.north})
            if (b->uts) std::free(b->uts);
        if (sstream) cudaStreamDestroy(sstream);
        if (ev_state) cudaEventDestroy(ev_state);
        if (ev_stats) cudaEventDestroy(ev_stats);
        if (own_stream && stream) cudaStreamDestroy(stream);
        (void)cudaGetLastError();   // teardown has no caller to report to; leave no stale error behind
    }

    template <typename T>
    int dalloc(T*& ptr, size_t count) {
        void* q = nullptr;
        CEL_CUDA_TRY(cudaMalloc(&q, count * sizeof(T)));
        CEL_CUDA_TRY(cudaMemset(q, 0, count * sizeof(T)));
        allocs.push_back(q);
        ptr = static_cast<T*>(q);
        return CEL_OK;
    }

    int init(const cel_params& prm, const float* bathy, int bnx, int bny) {
        p = prm;
        for (cel_boundary* b : {&p.west, &p.east, &p.south, &p.north})
            if (b->type != CEL_BC_UTS) { b->uts = nullptr; b->n_uts = 0; }
        if (int st = log_validate(p.log, p.nx, p.ny, err)) return st;
        int st0 = make_setup(p, bathy, bnx, bny, hs, err);
        if (st0) return st0;
        int dev = 0;
        CEL_CUDA_TRY(cudaGetDevice(&dev));
        CEL_CUDA_TRY(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
        own_stream = true;
        CEL_CUDA_TRY(cudaStreamCreateWithFlags(&sstream, cudaStreamNonBlocking));
        CEL_CUDA_TRY(cudaEventCreateWithFlags(&ev_state, cudaEventDisableTiming));
        CEL_CUDA_TRY(cudaEventCreateWithFlags(&ev_stats, cudaEventDisableTiming));
        c = make_consts(p, hs, hs.NX);
        ntex = size_t(hs.NX) * hs.NY;
        for (float4** t : {&st[0], &st[1], &st[2], &H, &U, &V, &AUX1, &AUX2, &BOT, &STRIP, &ABCx, &ABCy})
            if (int e = dalloc(*t, ntex)) return e;
        for (int k = 0; k < 4; ++k) {
            if (int e = dalloc(GRAD[k], ntex)) return e;
            if (int e = dalloc(FG[k], ntex)) return e;
        }
        if (int e = init_solve()) return e;
        {
            std::vector<float4> b(ntex);
            for (size_t i = 0; i < ntex; ++i) b[i] = make_float4(hs.BY[i], hs.BX[i], hs.BA[i], 0.f);
            CEL_CUDA_TRY(cudaMemcpy(BOT, b.data(), ntex * sizeof(float4), cudaMemcpyHostToDevice));
        }
        {   // irregular-wave component table: sides N, E, S, W back to back
            std::vector<float4> wv;
            const cel_boundary* sides[4] = {&p.north, &p.east, &p.south, &p.west};
            for (int s = 0; s < 4; ++s) {
                wave_off[s] = int(wv.size());
                if (sides[s]->type == CEL_BC_IRREGULAR)
                    for (int k = 0; k < sides[s]->n_waves; ++k)
                        wv.push_back(make_float4(float(sides[s]->waves[k][0]), float(sides[s]->waves[k][1]),
                                                 float(sides[s]->waves[k][2]), float(sides[s]->waves[k][3])));
            }
            if (wv.empty()) wv.push_back(make_float4(0, 0, 0, 0));
            if (int e = dalloc(WAVES, wv.size())) return e;
            CEL_CUDA_TRY(cudaMemcpy(WAVES, wv.data(), wv.size() * sizeof(float4), cudaMemcpyHostToDevice));
            // UTS tables stay on the host (timeSeriesHelper interpolates on the host)
            for (cel_boundary* b : {&p.west, &p.east, &p.south, &p.north}) {
                if (b->type == CEL_BC_UTS && b->n_uts > 0) {
                    double* copy = static_cast<double*>(std::malloc(sizeof(double) * 4 * b->n_uts));
                    std::memcpy(copy, b->uts, sizeof(double) * 4 * b->n_uts);
                    b->uts = copy;
                }
            }
        }
        const int nb = std::max(1, (hs.nx / 4) * (hs.ny / 4));
        if (int e = dalloc(blocks, size_t(nb) * 9)) return e;
        if (int e = dalloc(dstats, 16)) return e;
        stats_ctas = std::min(STATS_CTAS, (((hs.nx + 3) / 4) * ((hs.ny + 3) / 4) * 16 + STATS_THREADS - 1) / STATS_THREADS);
        if (int e = dalloc(spart, size_t(stats_ctas) * 11)) return e;
        if (int e = dalloc(sdone, 1)) return e;
        if (int e = init_boundary()) return e;
        // the set-up copies and memsets above ran on the legacy stream, which the engine's
        // non-blocking stream does not wait for: finish them
        CEL_CUDA_TRY(cudaDeviceSynchronize());
        return remesh();
    }

    // Work items of the one-launch boundary, where the domain's sides allow it.
    int init_boundary() {
        const cel_boundary* sides[4] = {&p.north, &p.east, &p.south, &p.west};
        int type[4], width[4];
        for (int s = 0; s < 4; ++s) { type[s] = sides[s]->type; width[s] = sides[s]->width; }
        planned = plan_boundary(hs.nx, hs.ny, type, width, regions);
        if (!planned) return CEL_OK;
        std::vector<int2> items;
        for (int k = 4; k < BND_REGIONS; ++k)
            if (regions[k].x1 > regions[k].x0 && regions[k].y1 > regions[k].y0) items.push_back(make_int2(k, 0));
        for (int k = 0; k < 4; ++k) {
            const int n = std::max(0, regions[k].x1 - regions[k].x0) * std::max(0, regions[k].y1 - regions[k].y0);
            for (int t = 0; t < n; t += 256) items.push_back(make_int2(k, t));
        }
        nbitems = int(items.size());
        if (int e = dalloc(bitems, std::max<size_t>(items.size(), 1))) return e;
        if (nbitems) CEL_CUDA_TRY(cudaMemcpy(bitems, items.data(), items.size() * sizeof(int2), cudaMemcpyHostToDevice));
        return CEL_OK;
    }

    // Level tables of the cyclic reduction and, once, the room for them.
    int init_solve() {
        tall = hs.nx <= CR_TALL_COLS && hs.ny >= CR_TALL_ROWS;
        const int cols = tall ? 1 : CR_COLS;
        auto levels = [&](const std::vector<int>& len, bool rows, int systems) {
            CrLevels L{};
            L.K = int(len.size());
            L.tail = L.K;
            size_t ko = 0, so = 0;
            for (int k = 0; k < L.K; ++k) {
                L.len[k] = len[k];
                L.off[k] = L.total;
                if (k > 0 || rows) L.total += len[k] + 1;   // one zero past a level's end
                L.koff[k] = ko;
                L.soff[k] = so;
                if (k > 0) ko += size_t(len[k]) * systems;
                so += size_t((len[k] + 1) / 2) * systems;
                if (k > 0 && L.tail == L.K && len[k] * (rows ? 1 : cols) <= 32) L.tail = k;
            }
            return std::make_pair(L, std::make_pair(ko, so));
        };
        const auto lx = levels(hs.lenx, true, hs.ny), ly = levels(hs.leny, false, hs.nx);
        solve.x = lx.first;
        solve.y = ly.first;
        if (int e = dalloc(K12x, lx.second.first)) return e;
        if (int e = dalloc(ACBx, lx.second.second)) return e;
        if (int e = dalloc(K12y, ly.second.first)) return e;
        if (int e = dalloc(ACBy, ly.second.second)) return e;
        solve.x.k12 = K12x; solve.x.acb = ACBx;
        solve.y.k12 = K12y; solve.y.acb = ACBy;
        const size_t bx = sizeof(float) * size_t(solve.x.total), by = sizeof(float) * size_t(solve.y.total) * cols;
        smem_x = bx <= CR_SMEM_MAX;
        smem_y = by <= CR_SMEM_MAX;
        smem_tall = tall ? by : 0;
        smem_cr = std::max(smem_x ? bx : 0, smem_y && !tall ? by : 0);
        solve.bands = tall ? 0 : (hs.nx + CR_COLS - 1) / CR_COLS;
        const size_t scratch = (smem_x ? 0 : size_t(hs.ny) * solve.x.total) +
                               (smem_y ? 0 : size_t(solve.bands) * CR_COLS * solve.y.total);
        if (scratch)
            if (int e = dalloc(solve.scratch, scratch)) return e;
        // the limit is the function's, not this engine's: set once to the most any engine asks for
        for (auto* k : {k_cr<true, true>, k_cr<true, false>, k_cr<false, true>, k_cr<false, false>, k_cr_tall})
            CEL_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(CR_SMEM_MAX)));
        // the allocations' clears ran on the legacy stream, which the engine's stream does not wait for
        CEL_CUDA_TRY(cudaDeviceSynchronize());
        return upload_solve();
    }

    // The solve's coefficients from the host's levels, on the engine's stream.  Packed on the device (on the
    // host it took 11 of the 89 ms of a 1001 x 777 engine's creation): levels above the first pass through H and U,
    // which every caller clears next.
    int upload_solve() {
        for (const bool rows : {true, false}) {
            const CrLevels& L = rows ? solve.x : solve.y;
            const auto& abc = rows ? hs.ABCx : hs.ABCy;
            const float4* prev = nullptr;
            for (int k = 0; k < L.K; ++k) {
                float4* cur = k == 0 ? (rows ? ABCx : ABCy) : (k & 1) ? H : U;
                const size_t count = k == 0 ? ntex : abc[k].size();
                if (count > ntex) { err = "a cyclic reduction level is larger than the domain"; return CEL_ERR_CUDA; }
                CEL_CUDA_TRY(cudaMemcpyAsync(cur, abc[k].data(), count * sizeof(float4), cudaMemcpyHostToDevice, stream));
                const int n = rows ? hs.ny : hs.nx, len = L.len[k];
                const size_t total = size_t(len) * n;
                if (total)
                    k_pack_level<<<unsigned((total + 255) / 256), 256, 0, stream>>>(
                        prev, cur, rows, n, len, k > 0 && rows ? L.len[k - 1] + 4 : 0, hs.NX, (rows ? K12x : K12y) + L.koff[k],
                        (rows ? ACBx : ACBy) + L.soff[k]);
                CEL_CUDA_TRY(cudaGetLastError());
                prev = cur;
            }
        }
        CEL_CUDA_TRY(cudaStreamSynchronize(stream));   // before the host copies go out of scope
        return CEL_OK;
    }

    int remesh() override {
        if (!terrain.empty()) {   // the bathymetry changed since creation: rebuild from the new grid
            HostSetup fresh;
            if (int st0 = make_setup(p, terrain.data(), terrain_nx, terrain_ny, fresh, err)) return st0;
            hs = fresh;
            if (int st0 = upload_solve()) return st0;
            // on the engine's stream, finished before the host copy goes out of scope
            std::vector<float4> b(ntex);
            for (size_t i = 0; i < ntex; ++i) b[i] = make_float4(hs.BY[i], hs.BX[i], hs.BA[i], 0.f);
            CEL_CUDA_TRY(cudaMemcpyAsync(BOT, b.data(), ntex * sizeof(float4), cudaMemcpyHostToDevice, stream));
            CEL_CUDA_TRY(cudaStreamSynchronize(stream));
        }
        std::vector<float4> s(ntex);
        for (size_t i = 0; i < ntex; ++i) s[i] = make_float4(hs.ic[3 * i], hs.ic[3 * i + 1], hs.ic[3 * i + 2], 0.f);
        CEL_CUDA_TRY(cudaMemcpyAsync(st[0], s.data(), ntex * sizeof(float4), cudaMemcpyHostToDevice, stream));
        CEL_CUDA_TRY(cudaMemcpyAsync(st[1], s.data(), ntex * sizeof(float4), cudaMemcpyHostToDevice, stream));
        for (float4* t : {H, U, V, AUX1, AUX2, GRAD[0], GRAD[1], GRAD[2], GRAD[3]})
            CEL_CUDA_TRY(cudaMemsetAsync(t, 0, ntex * sizeof(float4), stream));
        for (float2* t : FG) CEL_CUDA_TRY(cudaMemsetAsync(t, 0, ntex * sizeof(float2), stream));
        CEL_CUDA_TRY(cudaStreamSynchronize(stream));
        sch.reset(p);
        sim_idx = 0; cur_i = 0; old_i = 0; oldold_i = 1; scratch_i = 2; spare_i = 3; pred_i = 3;
        for (int& u : uts_iter) u = 1;
        faces_pending = faces_stored = false;
        return CEL_OK;
    }

    void uts_value(const cel_boundary& b, int side, float t, float out[3]) {
        // timeSeriesHelper (engine.cpp:1882-1904), with float arithmetic
        out[0] = out[1] = out[2] = 0.f;
        const int n = b.n_uts;
        int& it = uts_iter[side];
        while (it < n && float(b.uts[4 * it]) < t) ++it;
        if (it >= n) return;
        const float t0 = float(b.uts[4 * (it - 1)]), t1 = float(b.uts[4 * it]);
        const float m = (t - t0) / (t1 - t0);
        for (int q = 0; q < 3; ++q) {
            const float v0 = float(b.uts[4 * (it - 1) + q + 1]), v1 = float(b.uts[4 * it + q + 1]);
            out[q] = v0 + (v1 - v0) * m;
        }
    }

    // One side's settings at this pass; false if it has no texels.
    bool boundary_args(int side, BArgs& a) {
        const cel_boundary& b = side == 0 ? p.north : side == 1 ? p.east : side == 2 ? p.south : p.west;
        const int NX = hs.NX, NY = hs.NY;
        int x0, x1, y0, y1;
        if (side == 0) { x0 = 0; x1 = NX; y0 = NY - b.width; y1 = NY; }
        else if (side == 1) { x0 = NX - b.width; x1 = NX; y0 = 0; y1 = NY; }
        else if (side == 2) { x0 = 0; x1 = NX; y0 = 0; y1 = b.width; }
        else { x0 = 0; x1 = b.width; y0 = 0; y1 = NY; }
        x0 = std::max(x0, 0); y0 = std::max(y0, 0); x1 = std::min(x1, NX); y1 = std::min(y1, NY);
        a = BArgs{};
        if (x1 <= x0 || y1 <= y0) return false;
        a.side = side; a.type = b.type; a.width = b.width;
        a.sea_level = float(b.sea_level); a.amp = float(b.amplitude); a.period = float(b.period);
        a.theta = float(b.theta);
        a.n_waves = b.type == CEL_BC_IRREGULAR ? b.n_waves : 0;
        const int Kn = (side == 0 || side == 2) ? hs.Ky : hs.Kx;
        a.nleaf = 1 << (Kn - 1);
        a.waves = WAVES + wave_off[side];
        a.t = sch.total_time;
        a.dt = sch.dt;
        if (b.type == CEL_BC_UTS) {
            float v[3];
            uts_value(b, side, sch.total_time, v);
            a.uts_eta = v[0]; a.uts_hu = v[1]; a.uts_hv = v[2];
        }
        a.x0 = x0; a.y0 = y0; a.sw = x1 - x0; a.sh = y1 - y0;
        return true;
    }

    // boundaries East, North, West, South (engine.cpp:1342-1438)
    void boundaries(float4* stt) {
        if (planned) {
            BoundaryArgs a{};
            for (int side : {1, 0, 3, 2}) boundary_args(side, a.side[side]);
            std::copy(regions, regions + BND_REGIONS, a.region);
            if (nbitems == 0) return;
            TimedLaunch tl(&tm, stream, "plain_boundary");
            k_boundary_all<<<nbitems, 256, 0, stream>>>(stt, BOT, bitems, a, c);
            return;
        }
        for (int side : {1, 0, 3, 2}) {
            BArgs a;
            if (!boundary_args(side, a)) continue;
            {
                TimedLaunch tl(&tm, stream, "plain_boundary");
                k_boundary<<<grid2(a.sw, a.sh), dim3(BX2, BY2), 0, stream>>>(stt, BOT, STRIP, a, c);
            }
            TimedLaunch tl(&tm, stream, "plain_strip_copy");
            k_strip_copy<<<grid2(a.sw, a.sh), dim3(BX2, BY2), 0, stream>>>(stt, STRIP, a.x0, a.y0, a.sw, a.sh, hs.NX);
        }
    }

    int run_stats_kernels(cudaStream_t s) {
        (void)cudaGetLastError();
        {
            TimedLaunch tl(&tm, s, "plain_stats");
            k_stats<<<stats_ctas, STATS_THREADS, 0, s>>>(st[sim_idx], BOT, blocks, c, spart, sdone, dstats);
        }
        CEL_CUDA_TRY(cudaGetLastError());
        return CEL_OK;
    }
    int join_stats() {
        if (!stats_pending) return CEL_OK;
        stats_pending = false;
        CEL_CUDA_TRY(cudaStreamWaitEvent(stream, ev_stats, 0));
        return CEL_OK;
    }

    void finish_stats(const double* v, float cfl_used, cel_stats* o) {
        const double DENSITY = 1000;
        const double AREA = double(float(p.width) / float(hs.nx - 1) * float(p.length) / float(hs.ny - 1));
        const double g = double(c.g);
        o->mass = v[0] * DENSITY * AREA;
        o->potential_energy = v[1] * g * DENSITY * AREA;
        o->x_momentum = v[2] * DENSITY * AREA;
        o->y_momentum = v[3] * DENSITY * AREA;
        o->kinetic_energy = v[4] * 0.5 * DENSITY * AREA;
        o->total_energy = o->kinetic_energy + o->potential_energy;
        o->max_speed = std::sqrt(v[5]);
        o->max_depth = v[6];
        o->max_froude = std::sqrt(v[8] / g);
        o->cfl_rate = double(cfl_used);
        o->mass_full = v[9];
        o->health = v[10] != 0 ? CEL_ERR_NUMERIC : 0;
    }

    // resetTimestep: GetStats on the current state, then dt (engine.cpp:1536-1756)
    int reset_timestep(float, float, cel_stats* out) override {
        if (int e = join_stats()) return e;
        if (int e = run_stats_kernels(stream)) return e;
        double v[16];
        CEL_CUDA_TRY(cudaMemcpyAsync(v, dstats, sizeof(double) * 11, cudaMemcpyDeviceToHost, stream));
        CEL_CUDA_TRY(cudaStreamSynchronize(stream));
        const float cfl = sch.choose_dt(float(v[7]));
        if (out) {
            finish_stats(v, cfl, out);
            out->cfl_number = double(cfl * sch.dt);
            out->timestep = double(sch.dt);
            out->total_time = double(sch.total_time);
            out->time_scheme = sch.time_scheme;
        }
        last_stats_scheme = sch.time_scheme;
        last_stats_dt = sch.dt;
        last_stats_time = sch.total_time;
        return CEL_OK;
    }

    // resetTimestep without a host readback (fixed dt); adaptive dt needs the CFL on the host.
    int reset_timestep_device() {
        if (sch.adaptive) return reset_timestep(0.f, 0.f, nullptr);
        // On a stream of their own, beside the pass that follows (which reads the same state and writes
        // another one); that pass ends by waiting for them.  5 of 37 us a pass on 512 x 64 cells.
        if (int e = join_stats()) return e;
        CEL_CUDA_TRY(cudaEventRecord(ev_state, stream));
        CEL_CUDA_TRY(cudaStreamWaitEvent(sstream, ev_state, 0));
        if (int e = run_stats_kernels(sstream)) return e;
        CEL_CUDA_TRY(cudaEventRecord(ev_stats, sstream));
        stats_pending = true;
        sch.choose_dt(0.f);
        last_stats_scheme = sch.time_scheme;
        last_stats_dt = sch.dt;
        last_stats_time = sch.total_time;
        return CEL_OK;
    }

    int get_stats(cel_stats* out) override {
        if (int e = join_stats()) return e;
        double v[16];
        CEL_CUDA_TRY(cudaMemcpyAsync(v, dstats, sizeof(double) * 11, cudaMemcpyDeviceToHost, stream));
        CEL_CUDA_TRY(cudaStreamSynchronize(stream));
        finish_stats(v, float(v[7]), out);
        out->cfl_number = v[7] * double(last_stats_dt);
        out->timestep = double(last_stats_dt);
        out->total_time = double(last_stats_time);
        out->time_scheme = last_stats_scheme;
        return CEL_OK;
    }

    // timestep() (engine.cpp:849-1522): one pass
    int timestep() override {
        (void)cudaGetLastError();   // the launch checks below must see only this pass's launches
        if (!sch.initialized) { if (int e = reset_timestep(0.f, 0.f, nullptr)) return e; }
        const dim3 blk(BX2, BY2);
        int out_i;
        if (sch.time_scheme == CEL_SCHEME_CORRECTOR) {
            out_i = 3 - sim_idx - cur_i;
        } else {
            cur_i = sim_idx;
            out_i = (sim_idx + 1) % 3;
        }
        float4* old_state = st[sim_idx];
        float4* new_state = st[out_i];
        Pass3Args a{};
        a.st = old_state; a.bot = BOT; a.H = H; a.U = U; a.V = V; a.aux2 = AUX2; a.aux1 = AUX1;
        a.ABCx = ABCx; a.ABCy = ABCy;
        a.og = GRAD[old_i]; a.oog = GRAD[oldold_i]; a.ofg = FG[old_i]; a.oofg = FG[oldold_i];
        a.cur = st[cur_i]; a.pred = GRAD[pred_i]; a.fgpred = FG[pred_i];
        a.out = new_state; a.sgrad = GRAD[scratch_i]; a.sfg = FG[scratch_i];
        a.dt = sch.dt; a.dt_old = sch.dt_old; a.dt_old_old = sch.dt_old_old;
        a.decay = float(std::pow(double(std::fabs(c.whitewater_decay_rate)), double(sch.dt)));
        a.scheme = sch.time_scheme;
        {
            TimedLaunch tl(&tm, stream, "plain_pass123");
            if (faces_stored) k_pass123<true><<<grid2(hs.NX, hs.NY), blk, 0, stream>>>(a, c);
            else k_pass123<false><<<grid2(hs.NX, hs.NY), blk, 0, stream>>>(a, c);
        }
        const bool was_predictor = sch.is_predictor();
        // the implicit systems along x and y, in place (engine.cpp:1060-1217)
        {
            TimedLaunch tl(&tm, stream, "plain_cr");
            auto* k = smem_x ? (smem_y ? k_cr<true, true> : k_cr<true, false>) : (smem_y ? k_cr<false, true> : k_cr<false, false>);
            solve.st = new_state;
            if (tall) k_cr_tall<<<hs.nx, CR_TALL_THREADS, smem_tall, stream>>>(solve, c);
            k<<<hs.ny + solve.bands, CR_THREADS, smem_cr, stream>>>(solve, c);
        }
        boundaries(new_state);
        CEL_CUDA_TRY(cudaGetLastError());
        if (int e = join_stats()) return e;
        faces_pending = true;
        faces_stored = false;
        const bool book = sch.after_pass();
        if (book) {
            const int o = old_i, oo = oldold_i, s = scratch_i;
            old_i = s; oldold_i = o; scratch_i = oo;
        } else if (was_predictor) {   // the correctors read its derivatives and write elsewhere
            pred_i = scratch_i;
            std::swap(scratch_i, spare_i);
        }
        sim_idx = out_i;
        if (book && p.log.do_log && sch.last_count % p.log.log_step == 0) {
            // st_DumpToFile of the new state, with the time at the start of the step (engine.cpp:1488-1493)
            std::vector<float> host(ntex * 4);
            if (int e = get_state(host.data())) return e;
            if (int e = log_dump(p.log, host.data(), hs.nx, hs.ny, sch.last_start_time, log_elapsed, err)) return e;
        }
        return CEL_OK;
    }

    int timesteps(int n) override {
        for (int i = 0; i < n; ++i) {
            if (int e = reset_timestep_device()) return e;
            if (int e = timestep()) return e;
        }
        return CEL_OK;
    }

    int physical_steps(int n) override {
        for (int i = 0; i < n; ++i) {
            if (int e = reset_timestep_device()) return e;
            if (int e = timestep()) return e;
            while (sch.time_scheme == CEL_SCHEME_CORRECTOR) {
                if (int e = reset_timestep_device()) return e;
                if (int e = timestep()) return e;
            }
        }
        return CEL_OK;
    }

    int set_state(const float* rgba) override {
        CEL_CUDA_TRY(cudaMemcpyAsync(st[sim_idx], rgba, ntex * sizeof(float4), cudaMemcpyHostToDevice, stream));
        CEL_CUDA_TRY(cudaStreamSynchronize(stream));
        faces_pending = faces_stored = false;
        return CEL_OK;
    }
    int read_texture(const float4* t, float* rgba) {
        const size_t bytes = ntex * sizeof(float4);
        return rb.read(
            rgba, bytes, stream,
            [&](char* dst) { return cudaMemcpyAsync(dst, t, bytes, cudaMemcpyDeviceToHost, stream); },
            [&](size_t off, size_t n, char* slot) {
                return cudaMemcpyAsync(slot, reinterpret_cast<const char*>(t) + off, n, cudaMemcpyDeviceToHost, stream);
            },
            err);
    }
    int get_state(float* rgba) override {
        return read_texture(st[sim_idx], rgba);
    }
    int get_bottom(float* b3) override {
        for (size_t i = 0; i < ntex; ++i) { b3[3 * i] = hs.BY[i]; b3[3 * i + 1] = hs.BX[i]; b3[3 * i + 2] = hs.BA[i]; }
        return CEL_OK;
    }
    int get_aux(float* rgba) override {
        return read_texture(AUX1, rgba);
    }
    // newTerrainSettings -> fillTerrainTexture (engine.cpp:3313-3379): keep every texel's water depth
    // (w - BA_old + BA_new, in float as there), resample the bottom, clear both aux textures and
    // re-bootstrap.  The tridiagonal coefficients stay those of the old bottom until cel_remesh,
    // which rebuilds everything from the new grid (remesh re-creates the coefficient textures).
    int set_bathymetry(const float* z, int bnx, int bny) override {
        std::vector<float> host(ntex * 4);
        if (int e = get_state(host.data())) return e;
        for (size_t k = 0; k < ntex; ++k) host[4 * k] -= hs.BA[k];
        prepare_bottom(z, bnx, bny, hs.nx, hs.ny, float(p.width), float(p.length), hs);
        for (size_t k = 0; k < ntex; ++k) host[4 * k] += hs.BA[k];
        std::vector<float4> b(ntex);
        for (size_t i = 0; i < ntex; ++i) b[i] = make_float4(hs.BY[i], hs.BX[i], hs.BA[i], 0.f);
        CEL_CUDA_TRY(cudaMemcpyAsync(BOT, b.data(), ntex * sizeof(float4), cudaMemcpyHostToDevice, stream));
        CEL_CUDA_TRY(cudaMemcpyAsync(st[sim_idx], host.data(), ntex * sizeof(float4), cudaMemcpyHostToDevice, stream));
        CEL_CUDA_TRY(cudaMemsetAsync(AUX1, 0, ntex * sizeof(float4), stream));
        CEL_CUDA_TRY(cudaMemsetAsync(AUX2, 0, ntex * sizeof(float4), stream));
        CEL_CUDA_TRY(cudaStreamSynchronize(stream));
        terrain.assign(z, z + size_t(bnx) * bny);
        terrain_nx = bnx;
        terrain_ny = bny;
        faces_pending = faces_stored = false;
        return CEL_OK;
    }

    // the block sum of h comes from the latest GetStats (the state of the latest resetTimestep),
    // as the reference reads its GetStats staging texture
    int water_height(float x, float y, float* out) override {
        const float W = float(p.width), L = float(p.length);
        if (hs.nx < 4 || hs.ny < 4) { err = "getWaterHeight needs at least one 4x4 block"; return CEL_ERR_STATE; }
        if (!sch.initialized) { if (int e = reset_timestep(0.f, 0.f, nullptr)) return e; }
        if (int e = join_stats()) return e;
        int ix = 0, iy = 0;
        water_height_block(hs.nx, hs.ny, W, L, x, y, ix, iy);
        float sum_h = 0.f;
        CEL_CUDA_TRY(cudaMemcpyAsync(&sum_h, blocks + (size_t(iy) * (hs.nx / 4) + ix) * 9, sizeof(float),
                                     cudaMemcpyDeviceToHost, stream));
        CEL_CUDA_TRY(cudaStreamSynchronize(stream));
        *out = terrain_height(hs, W, L, x, y) + sum_h / 16.0f;
        return CEL_OK;
    }

    int add_solitary_wave(double Hh, double theta_deg, double xc, double yc) override {
        // the state texture is updated in place from a copy; faces are not rebuilt
        // (engine.cpp:2154-2219 leaves bootstrap_needed unchanged)
        float4* s = st[sim_idx];
        if (faces_pending && !faces_stored) {
            k_pass1<<<grid2(hs.nx + 2, hs.ny + 2), dim3(BX2, BY2), 0, stream>>>(s, BOT, AUX1, H, U, V, AUX2, c);
            faces_stored = true;
        }
        CEL_CUDA_TRY(cudaMemcpyAsync(STRIP, s, ntex * sizeof(float4), cudaMemcpyDeviceToDevice, stream));
        const float th = float(theta_deg) * CEL_PI_HOST / 180.0f;
        k_add_solitary<<<grid2(hs.nx + 2, hs.ny + 2), dim3(BX2, BY2), 0, stream>>>(STRIP, BOT, s, c, float(Hh), th,
                                                                                   float(xc), float(yc));
        CEL_CUDA_TRY(cudaGetLastError());
        CEL_CUDA_TRY(cudaStreamSynchronize(stream));
        return CEL_OK;
    }
    static constexpr float CEL_PI_HOST = 3.14159274101257324f;
    int set_stream(cudaStream_t s) override {
        CEL_CUDA_TRY(cudaStreamSynchronize(stream));
        if (own_stream) cudaStreamDestroy(stream);
        own_stream = (s == nullptr);
        if (own_stream) CEL_CUDA_TRY(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
        else stream = s;
        return CEL_OK;
    }
    int synchronize() override {
        CEL_CUDA_TRY(cudaStreamSynchronize(stream));
        return CEL_OK;
    }
    int set_tuning(int, int, int) override { return CEL_OK; }
    KernelTimer* timer() override { return &tm; }
    int nx() const override { return hs.nx; }
    int ny() const override { return hs.ny; }
};

}  // namespace

EngineIface* make_plain_engine(const cel_params& p, const float* bathy, int bnx, int bny, std::string& err) {
    auto* e = new PlainEngine();
    if (int s = e->init(p, bathy, bnx, bny)) {
        err = e->err;
        delete e;
        (void)s;
        return nullptr;
    }
    return e;
}

}  // namespace cel

// ---------------------------------------------------------------------------------------------
// Allocation-free statistics entry point.
//
// Some callers of this library must not allocate device memory at the moment they ask for the
// domain statistics: frame loops where the device-wide synchronisation of cudaMalloc / cudaFree
// would stall every other stream, and host applications whose device memory is entirely handed out
// by their own allocator.  cel_stats_noalloc computes the GetStats reduction and the FP64 volume of
// a state that the caller already keeps in device memory, using only the fixed scratch array below:
// the 4x4 block partials, the volume partials and the FP64 totals.  The array is reserved on every
// GPU that loads the library and stays there until the process exits.  All calls share it, so two
// calls whose work overlaps on the GPU (on different streams, or from different threads) race; run
// them one after another.
// ---------------------------------------------------------------------------------------------
namespace cel {
namespace {

constexpr int NOALLOC_MAX_BLOCKS = 65536;                  // 4x4 blocks: up to 1,048,576 cells
constexpr int NOALLOC_VOL_CTAS = 1184;                     // volume partials: 8 CTAs per SM of a B200
// block partials (9 floats each) | volume partials (2 doubles per CTA) | 16 doubles of totals
constexpr int NOALLOC_FLOATS = NOALLOC_MAX_BLOCKS * 9 + NOALLOC_VOL_CTAS * 4 + 32;
static __device__ __align__(256) float g_noalloc_scratch[NOALLOC_FLOATS];

// GetStats (compute.hlsl:1319-1378) reading the bottom in the public {BY, BX, BA} layout.
__global__ void k_getstats_b3(const float4* __restrict__ st, const float* __restrict__ b3, float* __restrict__ blocks,
                              SimConsts c) {
    const int bx = blockIdx.x * blockDim.x + threadIdx.x;
    const int by = blockIdx.y * blockDim.y + threadIdx.y;
    const int nbx = c.nx / 4, nby = c.ny / 4;
    if (bx >= nbx || by >= nby) return;
    float sh = 0, sb = 0, shu = 0, shv = 0, sk = 0, mu = 0, mh = 0, mc = 0, mf = 0;
    for (int j = 2; j < 6; ++j)
        for (int ii = 2; ii < 6; ++ii) {
            const size_t i = size_t(by * 4 + j) * c.NX + bx * 4 + ii;
            const float4 s = st[i];
            const float B = b3[3 * i + 2];
            const float h = fmaxf(0.f, s.x - B);
            const float cc = sqrtf(c.g * h);
            const float q = div_by_h(h, c.epsilon);
            const float u = q * s.y, v = q * s.z;
            sh += h; sb += h * (B + 0.5f * h); shu += s.y; shv += s.z;
            sk += (s.y * u + s.z * v);
            const float u2v2 = u * u + v * v;
            mu = fmaxf(mu, u2v2); mh = fmaxf(mh, h);
            mc = fmaxf(mc, (fabsf(u) + cc) * c.one_over_dx);
            mc = fmaxf(mc, (fabsf(v) + cc) * c.one_over_dy);
            mf = fmaxf(mf, u2v2 * q);
        }
    float* o = blocks + (size_t(by) * nbx + bx) * 9;
    o[0] = sh; o[1] = sb; o[2] = shu; o[3] = shv; o[4] = sk; o[5] = mu; o[6] = mh; o[7] = mc; o[8] = mf;
}

// FP64 volume of the interior cells (and the non-finite flag), one partial per CTA: CTA k sums a
// fixed interleaved share of the cells, so the totals do not depend on scheduling.
__global__ void __launch_bounds__(256) k_volume_b3(const float4* __restrict__ st, const float* __restrict__ b3,
                                                   SimConsts c, double* __restrict__ part) {
    __shared__ double sv[8];
    __shared__ int sb;
    if (threadIdx.x == 0) sb = 0;
    __syncthreads();
    double v = 0.0;
    int bad = 0;
    const int n = c.nx * c.ny;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const size_t i = size_t(k / c.nx + 2) * c.NX + (k % c.nx + 2);
        const float4 s = st[i];
        if (!isfinite(s.x) || !isfinite(s.y) || !isfinite(s.z)) bad = 1;
        v += fmax(0.0, double(s.x) - double(b3[3 * i + 2]));
    }
    for (int off = 16; off; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0) sv[threadIdx.x >> 5] = v;
    if (bad) sb = 1;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += sv[w];
        part[2 * blockIdx.x] = t;
        part[2 * blockIdx.x + 1] = sb ? 1.0 : 0.0;
    }
}

// One CTA: FP64 totals of the block partials and the volume partials; every output word is
// written on every call.
__global__ void k_reduce_b3(const float* __restrict__ blocks, int nb, const double* __restrict__ vol, int nvol,
                            double* __restrict__ out) {
    __shared__ double sm[10][32];
    __shared__ int bad_s;
    double v[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    int bad = 0;
    for (int k = threadIdx.x; k < nb; k += blockDim.x) {
        const float* b = blocks + size_t(k) * 9;
        for (int q = 0; q < 5; ++q) v[q] += double(b[q]);
        for (int q = 5; q < 9; ++q) v[q] = fmax(v[q], double(b[q]));
    }
    for (int k = threadIdx.x; k < nvol; k += blockDim.x) {
        v[9] += vol[2 * k];
        if (vol[2 * k + 1] != 0.0) bad = 1;
    }
    if (threadIdx.x == 0) bad_s = 0;
    __syncthreads();
    if (bad) bad_s = 1;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int q = 0; q < 10; ++q) {
        double x = v[q];
        for (int off = 16; off; off >>= 1) {
            const double y = __shfl_down_sync(0xffffffffu, x, off);
            x = (q >= 5 && q < 9) ? fmax(x, y) : x + y;
        }
        if (lane == 0) sm[q][wid] = x;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int nw = blockDim.x >> 5;
        for (int q = 0; q < 10; ++q) {
            double x = lane < nw ? sm[q][lane] : 0.0;
            for (int off = 16; off; off >>= 1) {
                const double y = __shfl_down_sync(0xffffffffu, x, off);
                x = (q >= 5 && q < 9) ? fmax(x, y) : x + y;
            }
            if (lane == 0) out[q] = x;
        }
        if (lane == 0) out[10] = bad_s ? 1.0 : 0.0;
    }
}

// Device address of the scratch array, looked up once per device (with that device current).
constexpr int NOALLOC_MAX_DEVICES = 64;
float* g_noalloc_ptr[NOALLOC_MAX_DEVICES] = {nullptr};   // guarded by g_noalloc_mutex
std::mutex g_noalloc_mutex;

}  // namespace

}  // namespace cel

extern "C" int cel_stats_noalloc(const float* d_state_rgba, const float* d_bottom_b3, const cel_params* p,
                                 void* cuda_stream, cel_stats* out) {
    using namespace cel;
    if (!d_state_rgba || !d_bottom_b3 || !p || !out) { set_error("null argument"); return CEL_ERR_ARG; }
    if (p->nx < 4 || p->ny < 4) { set_error("cel_stats_noalloc: nx and ny must be >= 4"); return CEL_ERR_ARG; }
    const long long nb = (long long)(p->nx / 4) * (p->ny / 4);
    if (nb > NOALLOC_MAX_BLOCKS) {
        set_error("cel_stats_noalloc: domain has " + std::to_string(nb) + " 4x4 blocks; the fixed scratch holds " +
                  std::to_string(NOALLOC_MAX_BLOCKS) + " (at most 1,048,576 interior cells)");
        return CEL_ERR_ARG;
    }
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) { set_error(std::string("cel_stats_noalloc: ") + cudaGetErrorString(e)); return CEL_ERR_CUDA; }
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) { set_error("cel_stats_noalloc: device index out of range"); return CEL_ERR_ARG; }
    float* blocks = nullptr;
    {
        // the array's device address on this device, resolved by the first call here (with the
        // device current) under a lock, so that concurrent first calls do not race
        std::lock_guard<std::mutex> lock(g_noalloc_mutex);
        if (!g_noalloc_ptr[dev]) {
            float* ptr = nullptr;
            e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_noalloc_scratch);
            if (e != cudaSuccess || !ptr) {
                set_error(std::string("cel_stats_noalloc: cudaGetSymbolAddress failed: ") + cudaGetErrorString(e));
                return CEL_ERR_CUDA;
            }
            g_noalloc_ptr[dev] = ptr;
        }
        blocks = g_noalloc_ptr[dev];
    }
    // volume partials after the block partials (byte offset 65,536 x 36, a multiple of 256), totals last
    double* vol = reinterpret_cast<double*>(blocks + size_t(NOALLOC_MAX_BLOCKS) * 9);
    double* totals = vol + 2 * NOALLOC_VOL_CTAS;
    HostSetup hs;
    hs.nx = p->nx; hs.ny = p->ny; hs.NX = p->nx + 4; hs.NY = p->ny + 4;
    hs.dx = float(p->width) / float(p->nx - 1);
    hs.dy = float(p->length) / float(p->ny - 1);
    {
        const float m = std::max(hs.dx, hs.dy);
        hs.eps = std::min(float(p->epsilon), m * m * m * m);
    }
    const SimConsts c = make_consts(*p, hs, hs.NX);
    cudaStream_t s = static_cast<cudaStream_t>(cuda_stream);
    const float4* st = reinterpret_cast<const float4*>(d_state_rgba);
    const int nbx = p->nx / 4, nby = p->ny / 4;
    k_getstats_b3<<<grid2(nbx, nby), dim3(BX2, BY2), 0, s>>>(st, d_bottom_b3, blocks, c);
    const int nvol = int(std::min<long long>(NOALLOC_VOL_CTAS, (p->nx * (long long)p->ny + 255) / 256));
    k_volume_b3<<<nvol, 256, 0, s>>>(st, d_bottom_b3, c, vol);
    k_reduce_b3<<<1, 1024, 0, s>>>(blocks, int(nb), vol, nvol, totals);
    e = cudaGetLastError();
    if (e != cudaSuccess) { set_error(std::string("cel_stats_noalloc: ") + cudaGetErrorString(e)); return CEL_ERR_CUDA; }
    double v[11];
    e = cudaMemcpyAsync(v, totals, sizeof(v), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) { set_error(std::string("cel_stats_noalloc: ") + cudaGetErrorString(e)); return CEL_ERR_CUDA; }
    const double DENSITY = 1000;
    const double AREA = double(float(p->width) / float(p->nx - 1) * float(p->length) / float(p->ny - 1));
    const double g = double(c.g);
    std::memset(out, 0, sizeof(*out));
    out->mass = v[0] * DENSITY * AREA;
    out->potential_energy = v[1] * g * DENSITY * AREA;
    out->x_momentum = v[2] * DENSITY * AREA;
    out->y_momentum = v[3] * DENSITY * AREA;
    out->kinetic_energy = v[4] * 0.5 * DENSITY * AREA;
    out->total_energy = out->kinetic_energy + out->potential_energy;
    out->max_speed = std::sqrt(v[5]);
    out->max_depth = v[6];
    out->cfl_rate = v[7];
    out->max_froude = std::sqrt(v[8] / g);
    out->mass_full = v[9];
    out->health = v[10] != 0 ? CEL_ERR_NUMERIC : 0;
    out->timestep = p->timestep;
    out->cfl_number = out->cfl_rate * double(float(p->timestep));
    return CEL_OK;
}

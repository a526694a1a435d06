// One launch per time step for elastic, VTI and acoustic-elastic grids.
//
// A launch advances every shot of a plan by one step.  Its CTAs (256 threads)
// take three kinds of work units, the boundary units first:
//   x-band     32 z cells of the 6 columns next to the left or right edge;
//   z-band     32 columns of the 6 rows next to the top or bottom edge;
//   interior   a window of 32 (z) x 16 (x) cells clear of the bands.
// Each unit performs the whole step of the reference time loop
// (src/cpp/we_op.cpp:667-871 elastic, :1640-1840 VTI, :2240-2530 the elastic
// grid of the acoustic-elastic propagator) with receivers, snapshots or the
// imaging condition, in the reference's single-precision operation order.
//
// Consecutive steps are chained by programmatic dependent launch: a CTA of
// step n+1 that finds a free slot while step n runs stages everything step n
// does not write (model, boundary closures, snapshots of the imaging
// condition) in shared memory before it waits for step n (griddepcontrol.wait).
// Fields and gradients are read after the wait and through L2 (.cg): a line of
// theirs may lie in L1 from before the wait.
#include <cuda_runtime.h>
#include "engine.h"
#include "sbp.cuh"
#include "snap.cuh"
#include "launch.h"

namespace fwi2d {

// (1, 1) and (-1, -1), set at run time: the multipliers of the packed sums (sbp.cuh add2)
static __constant__ float2 kMinus2;

constexpr int kFz = kFusedZ, kFx = kFusedX;      // interior window
constexpr int kFs = kFz + 8;                     // row stride of every staged array (floats)
constexpr int kFt = 256;                         // threads: a z-pair of the interior window each
constexpr int kFu = (kFx + 8) * kFs, kFw = (kFx + 4) * kFs, kFo = kFx * kFz;
constexpr int kFb = 10;                          // band units: samples staged along the normal
static_assert(kFt == kFz / 2 * kFx, "one z-pair per thread");

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// 16-byte asynchronous copy through L2; zeros when !ok (nothing is read then)
__device__ __forceinline__ void cp16(float *dst, const float *src, bool ok)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(ok ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ---- packed arithmetic beyond sbp.cuh ---------------------------------------
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
    float2 r;
    asm("{\n .reg .b64 pa, pb, pc, pd;\n mov.b64 pa, {%2, %3};\n mov.b64 pb, {%4, %5};\n mov.b64 pc, {%6, %7};\n"
        " fma.rn.f32x2 pd, pa, pb, pc;\n mov.b64 {%0, %1}, pd;\n}\n"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}
// a - b, rounded once, with nothing left to fuse (add2 with the multiplier -1)
__device__ __forceinline__ float2 dif2(float2 a, float2 b) { return fma2(b, kMinus2, a); }
// lane by lane, for operands whose lanes do not sit in one register pair
__device__ __forceinline__ float2 mulx(float ax, float ay, float2 b) { return make_float2(ax * b.x, ay * b.y); }

// x / b rounded to nearest for r = 1/b rounded to nearest: two correction
// steps of Markstein's division (IBM J. Res. Dev. 34, 1990); the first makes the
// quotient faithful, the second rounds it correctly.  Exact while neither the
// quotient nor the remainder leaves the normal range: |x| in [2^-100, 2^100]
// and b in [2^-20, 2^20]; other operands take the divide (r = 0 marks such a b).
constexpr float kDivLo = 7.888609052210118e-31f, kDivHi = 1.2676506002282294e30f;
__device__ __forceinline__ float div_by(float x, float b, float r)
{
    const float a = fabsf(x);
    if (a >= kDivLo && a <= kDivHi && r > 0.f) {
        float q = x * r;
        q = fmaf(fmaf(-q, b, x), r, q);
        return fmaf(fmaf(-q, b, x), r, q);
    }
    return x / b;
}

// both components of a z-pair over the pair's densities
__device__ __forceinline__ void div_pairs(float2 &x0, float2 &x1, float2 b, float2 r)
{
    const float hi = fmaxf(fmaxf(fabsf(x0.x), fabsf(x0.y)), fmaxf(fabsf(x1.x), fabsf(x1.y)));
    const float lo = fminf(fminf(fabsf(x0.x), fabsf(x0.y)), fminf(fabsf(x1.x), fabsf(x1.y)));
    if (lo >= kDivLo && hi <= kDivHi && fminf(r.x, r.y) > 0.f) {
        const float2 nb = make_float2(-b.x, -b.y);
        float2 q0 = mul2(x0, r), q1 = mul2(x1, r);
        q0 = fma2(fma2(q0, nb, x0), r, q0);
        q1 = fma2(fma2(q1, nb, x1), r, q1);
        x0 = fma2(fma2(q0, nb, x0), r, q0);
        x1 = fma2(fma2(q1, nb, x1), r, q1);
    } else if (hi == 0.f && fminf(b.x, b.y) > 0.f) {
        return;   // 0 / b for both components: the zeros keep their signs
    } else {
        x0 = make_float2(x0.x / b.x, x0.y / b.y);
        x1 = make_float2(x1.x / b.x, x1.y / b.y);
    }
}

// Interior weights of Dxx_var/Dzz_var (kC2, upload_sbp_tables) as literals.
// The products with 1/2 and 1/8 are exact, so an fma of them rounds once, as
// the separate sum does.
#define KC_S6 0.16666667163372040f
__device__ __forceinline__ Brk2 brackets2(float2 fm2, float2 fm1, float2 f0, float2 fp1, float2 fp2)
{
    const float2 s6 = bc2(KC_S6), h = bc2(0.5f), e = bc2(-0.125f);
    const float2 sm2 = mul2(s6, fm2), sp2 = mul2(s6, fp2), sm1 = mul2(s6, fm1), sp1 = mul2(s6, fp1);
    Brk2 b;
    b.b0 = add2(add2(mul2(bc2(kC2[0]), f0), mul2(bc2(kC2[1]), add2(fm1, fp1))), mul2(bc2(kC2[2]), add2(fm2, fp2)));
    b.bm1 = add2(fma2(h, f0, fma2(h, fm1, sm2)), sp1);
    b.bp1 = add2(fma2(h, f0, fma2(h, fp1, sp2)), sm1);
    b.bm2 = fma2(e, f0, fma2(e, fm2, sm1));
    b.bp2 = fma2(e, f0, fma2(e, fp2, sp1));
    return b;
}

// b0 u0 + bm1 um1 + bp1 up1 + bm2 um2 + bp2 up2 along z for the pair `mid`
// with its neighbours lo, hi: um1 = (lo.y, mid.x), up1 = (mid.y, hi.x)
__device__ __forceinline__ float2 sum_z(const Brk2 &b, float2 lo, float2 mid, float2 hi)
{
    const float2 t1 = mulx(lo.y, mid.x, b.bm1), t2 = mulx(mid.y, hi.x, b.bp1);
    return add2(add2(add2(add2(mul2(b.b0, mid), t1), t2), mul2(b.bm2, lo)), mul2(b.bp2, hi));
}
__device__ __forceinline__ float2 sum_x(const Brk2 &b, float2 um2, float2 um1, float2 u0, float2 up1, float2 up2)
{
    return add2(add2(add2(add2(mul2(b.b0, u0), mul2(b.bm1, um1)), mul2(b.bp1, up1)), mul2(b.bm2, um2)),
                mul2(b.bp2, up2));
}
// first derivatives (sbp.cuh d1s) of loaded samples along x and z
__device__ __forceinline__ float2 der_x(float2 um2, float2 um1, float2 up1, float2 up2, float s)
{
    return mul2(bc2(s), add2(mul2(bc2(kC1[0]), dif2(up1, um1)), mul2(bc2(kC1[1]), dif2(up2, um2))));
}
__device__ __forceinline__ float2 der_z(float2 lo, float2 mid, float2 hi, float s)
{
    const float2 d = make_float2(mid.y - lo.y, hi.x - mid.x);
    return mul2(bc2(s), add2(mul2(bc2(kC1[0]), d), mul2(bc2(kC1[1]), dif2(hi, lo))));
}

// ---------------------------------------------------------------------------
// shared-memory layouts (floats)
// ---------------------------------------------------------------------------
// Interior: curr with a 4-cell halo (U), everything else with a 2-cell halo
// along x and the same row stride, so that one index serves all arrays.  P, R,
// S: the products lambda (ux_x + uz_z), mu ux_z and mu uz_x of the mixed terms,
// formed once per cell (VTI: P = tmp_x and P1 = tmp_z; acoustic-elastic: P =
// lambda ux_x, P1 = lambda uz_z).  O: the window's own cells, 32 x 16 each.
template <bool VTI, bool GRAD, bool AE>
struct InLayout {
    static constexpr int U0 = 0, U1 = kFu, MU = 2 * kFu, Q = MU + kFw, P = Q + kFw, R = P + kFw, S = R + kFw;
    static constexpr int P1 = S + kFw, LB = P1 + (VTI || AE ? kFw : 0), LC = LB + (VTI ? kFw : 0);
    static constexpr int LA = LC + (VTI ? kFw : 0), F0 = LA + (VTI ? kFw : 0), F1 = F0 + (GRAD ? kFw : 0);
    static constexpr int O = F1 + (GRAD ? kFw : 0);
    // own-cell arrays
    static constexpr int PV0 = O, PV1 = O + kFo, RHO = O + 2 * kFo, IR = O + 3 * kFo, G0 = O + 4 * kFo;
    static constexpr int FP0 = G0 + (GRAD ? 3 * kFo : 0), FM0 = FP0 + (GRAD ? 2 * kFo : 0);
    static constexpr int E = FM0 + (GRAD ? 2 * kFo : 0);   // VTI imaging: eps, v2, v3
    static constexpr int RED = E + (VTI && GRAD ? 3 * kFo : 0);
    static constexpr int FLOATS = RED + 8;
};

// Bands: [10 normal samples][40 tangential samples] per array, then the
// closure coefficients of the owned rows, [6][8][32].
template <bool VTI, bool GRAD>
struct BandLayout {
    static constexpr int A = kFb * kFs, CL = 6 * 8 * 32;
    static constexpr int U0 = 0, U1 = A, MU = 2 * A, Q = 3 * A, T0 = 4 * A, CZ = 5 * A, BX = 6 * A, T1 = 7 * A;
    static constexpr int LB = 8 * A, LC = LB + (VTI ? A : 0), LA = LC + (VTI ? A : 0);
    static constexpr int F0 = LA + (VTI ? A : 0), F1 = F0 + (GRAD ? A : 0), C0 = F1 + (GRAD ? A : 0);
    static constexpr int C1 = C0 + CL;                     // VTI x bands: closure of (1+2eps)2mu
    static constexpr int RED = C1 + (VTI ? CL : 0);
    static constexpr int FLOATS = RED + 8;
};

template <bool VTI, bool GRAD, bool AE>
constexpr size_t fused_bytes()
{
    return sizeof(float) * (InLayout<VTI, GRAD, AE>::FLOATS > BandLayout<VTI, GRAD>::FLOATS
                                ? InLayout<VTI, GRAD, AE>::FLOATS
                                : BandLayout<VTI, GRAD>::FLOATS);
}

struct FusedArgs {
    const ShotDev *shots;
    const TileRef *xb;
    const BandRef *zb;
    const TileRef *in;
    int nxb, nzb;
    ModelDev M;
    StepConst C;
    int it, flags;
    float dtg;
};

// max |next| of a CTA for the scale of the next 16-bit snapshot
__device__ __forceinline__ void block_amax(float m, float *red, unsigned *dst)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        m = red[0];
#pragma unroll
        for (int w = 1; w < kFt / 32; w++) m = fmaxf(m, red[w]);
        if (m > 0.f) atomicMax(dst, __float_as_uint(m));
    }
}

// Four snapshot samples (index a multiple of 4) as FP32.
__device__ __forceinline__ float4 snap_load4(const void *base, long long idx, int prec, float inv)
{
    const float2 a = snap_load2(base, idx, prec, inv), b = snap_load2(base, idx + 2, prec, inv);
    return make_float4(a.x, a.y, b.x, b.y);
}

// Density term of the imaging condition at one cell, in the reference's mixed
// precision: k = 0 the first snapshot, `last` the last one.
__device__ __forceinline__ float density_term(float g, double wdt, int k, int last, float a0, float a1, float f0, float f1,
                                              float fp0, float fp1, float fm0, float fm1)
{
    float s;
    if (k > 0 && k < last) s = a0 * (fp0 - 2 * f0 + fm0) + a1 * (fp1 - 2 * f1 + fm1);
    else if (k == 0) s = a0 * (fp0 - f0) + a1 * (fp1 - f1);
    else s = a0 * (-f0 + fm0) + a1 * (-f1 + fm1);
    return (float)((double)g + wdt * (double)s);
}

// ---------------------------------------------------------------------------
// Interior window.  Thread t owns the z-pair 2 (t & 15) of column t >> 4.
// Measured on B200, see launch_fused_step.
// ---------------------------------------------------------------------------
template <bool VTI, bool GRAD, bool AE>
__device__ __forceinline__ void fused_interior(const FusedArgs &A, const TileRef tr, float *sm)
{
    using L = InLayout<VTI, GRAD, AE>;
    const ModelDev &M = A.M;
    const StepConst &C = A.C;
    const int t = threadIdx.x, it = A.it;
    const ShotDev *__restrict__ Sp = A.shots + tr.shot;
    const int nt = Sp->nt, nx = Sp->nx, ldz = Sp->ldz;
    const int nxz = nx * ldz;
    const int prec = C.snap_prec;
    const long long mofs = (long long)Sp->x0 * ldz;   // the model has the shots' pitch
    const int itf = GRAD ? (nt - 1 - (it + 1)) / C.sub : 0;
    const bool do_grad = GRAD && it < nt - 1 && ((nt - 1 - (it + 1)) % C.sub == 0) && (!AE || itf != 0);
    const int last = nt / C.sub;
    const int xr = t / 10, xq = 4 * (t - 10 * xr);    // staged row and sample of this thread's copies
    const int orow = (t >> 3) & 15, oq = 4 * (t & 7); // the same for the own-cell arrays (two per pass)

    // ---- what no step writes: coefficients, densities, snapshots
    if (t < (kFx + 4) * 10) {
        const int gx = tr.wx0 - 2 + xr, gz = tr.wz0 - 4 + xq;
        const bool ok = gx < nx && gz < ldz;
        const long long o = mofs + (ok ? (long long)gx * ldz + gz : 0);
        const int s = xr * kFs + xq;
        cp16(sm + L::MU + s, M.p1 + o, ok);
        cp16(sm + L::Q + s, (VTI ? M.fxx : M.p0) + o, ok);
        if (VTI) {
            cp16(sm + L::LB + s, M.lbis + o, ok);
            cp16(sm + L::LC + s, M.c13 + o, ok);
            cp16(sm + L::LA + s, M.p0 + o, ok);
        }
        if (GRAD && do_grad) {
            const long long so = (long long)itf * Sp->snap_slot + (ok ? (long long)gx * ldz + gz : 0);
            if (prec == SNAP_FP32) {
                cp16(sm + L::F0 + s, (const float *)Sp->snap + so, ok);
                cp16(sm + L::F1 + s, (const float *)Sp->snap + so + nxz, ok);
            } else if (ok) {
                const float inv = 1.f / snap_scale(Sp->snap_amax, itf);
                *reinterpret_cast<float4 *>(sm + L::F0 + s) = snap_load4(Sp->snap, so, prec, inv);
                *reinterpret_cast<float4 *>(sm + L::F1 + s) = snap_load4(Sp->snap, so + nxz, prec, inv);
            }
        }
    }
    const int ogx = tr.wx0 + orow, ogz = tr.wz0 + oq;
    const bool ook = ogx < nx && ogz < ldz;
    const long long oc = ook ? (long long)ogx * ldz + ogz : 0;
    const int os = (t >> 7) * kFo + orow * kFz + oq;
    cp16(sm + L::RHO + os, ((t >> 7) ? M.irho : M.p2) + mofs + oc, ook);
    if (GRAD && do_grad) {
        const long long oo = oc + (t >> 7 ? nxz : 0);
        auto own_snap = [&](int dst, int k, bool have) {
            const long long so = (long long)k * Sp->snap_slot + oo;
            if (prec == SNAP_FP32 || !have) {
                cp16(sm + dst + os, (const float *)Sp->snap + (have ? so : 0), ook && have);
            } else if (ook) {
                const float inv = 1.f / snap_scale(Sp->snap_amax, k);
                *reinterpret_cast<float4 *>(sm + dst + os) = snap_load4(Sp->snap, so, prec, inv);
            }
        };
        own_snap(L::FP0, itf + 1, itf + 1 <= last);
        own_snap(L::FM0, itf - 1, itf > 0);
        if (VTI) {
            cp16(sm + L::E + os, ((t >> 7) ? M.gv2 : M.eps) + mofs + oc, ook);
            if (t < 128) cp16(sm + L::E + 2 * kFo + os, M.gv3 + mofs + oc, ook);
        }
    }
    const int tx = t >> 4, pz = 2 * (t & 15);
    const int gx = tr.wx0 + tx, gz = tr.wz0 + pz;
    const bool ownx = gx >= tr.ox0 && gx < tr.ox1;
    const bool own0 = ownx && gz >= tr.oz0 && gz < tr.oz1, own1 = ownx && gz + 1 >= tr.oz0 && gz + 1 < tr.oz1;
    float2 tzv = make_float2(0.f, 0.f);
    float txv = 0.f;
    if (own0 || own1) {
        tzv = *reinterpret_cast<const float2 *>(Sp->tz + gz);
        txv = Sp->tx[gx];
    }
    const int e0 = Sp->inj_off[tr.unit], e1 = Sp->inj_off[tr.unit + 1];
    const float *curr = Sp->u[(it + 1) & 1];
    float *pn = Sp->u[it & 1];   // prev in, next out

    pdl_wait();
    pdl_launch();
    if (it >= nt - 1) {
        cp_wait();
        return;
    }

    // ---- fields and, in the adjoint, the gradient
    if (t < (kFx + 8) * 10) {
        const int x = tr.wx0 - 4 + xr, z = tr.wz0 - 4 + xq;
        const bool ok = x < nx && z < ldz;
        const long long o = ok ? (long long)x * ldz + z : 0;
        const int s = xr * kFs + xq;
        cp16(sm + L::U0 + s, curr + o, ok);
        cp16(sm + L::U1 + s, curr + nxz + o, ok);
    }
    cp16(sm + L::PV0 + os, pn + (t >> 7 ? nxz : 0) + oc, ook);
    if (GRAD && do_grad) {
        cp16(sm + L::G0 + os, Sp->grad + (t >> 7 ? nxz : 0) + oc, ook);
        if (t < 128) cp16(sm + L::G0 + 2 * kFo + os, Sp->grad + 2 * (long long)nxz + oc, ook);
    }
    cp_wait();
    __syncthreads();

    const float *U0 = sm + L::U0 + 2 * kFs, *U1 = sm + L::U1 + 2 * kFs;   // indexed as the 2-halo arrays
    const float *MU = sm + L::MU, *Q = sm + L::Q;
    float *P = sm + L::P, *R = sm + L::R, *S = sm + L::S, *P1 = sm + L::P1;

    // products of the mixed terms at one pair from its strains
    auto mixed = [&](int i, float2 exx, float2 ezz) {
        if (VTI) {
            const float2 lb = ld2(sm + L::LB, i), lc = ld2(sm + L::LC, i), la = ld2(sm + L::LA, i);
            *reinterpret_cast<float2 *>(P + i) = add2(mul2(lb, exx), mul2(lc, ezz));
            *reinterpret_cast<float2 *>(P1 + i) = add2(mul2(la, ezz), mul2(lc, exx));
        } else if (AE) {
            const float2 q = ld2(Q, i);
            *reinterpret_cast<float2 *>(P + i) = mul2(exx, q);
            *reinterpret_cast<float2 *>(P1 + i) = mul2(ezz, q);
        } else {
            *reinterpret_cast<float2 *>(P + i) = mul2(add2(exx, ezz), ld2(Q, i));
        }
    };

    // ---- halo pairs: 4 columns beside the window (P, R), 2 x 16 pairs above and below it (P, S)
    if (t < 96) {
        const bool side = t < 64;
        const int r = t >> 4;
        int i;
        if (side) i = (r < 2 ? r : r + kFx) * kFs + 4 + pz;
        else i = (2 + ((t - 64) >> 1)) * kFs + 2 + ((t & 1) ? kFz + 2 : 0);
        const float2 exx = der_x(ld2(U0, i - 2 * kFs), ld2(U0, i - kFs), ld2(U0, i + kFs), ld2(U0, i + 2 * kFs), C.sdx);
        const float2 ezz = der_z(ld2(U1, i - 2), ld2(U1, i), ld2(U1, i + 2), C.sdz);
        mixed(i, exx, ezz);
        const float2 m = ld2(MU, i);
        if (side)
            *reinterpret_cast<float2 *>(R + i) = mul2(der_z(ld2(U0, i - 2), ld2(U0, i), ld2(U0, i + 2), C.sdz), m);
        else
            *reinterpret_cast<float2 *>(S + i) =
                mul2(der_x(ld2(U1, i - 2 * kFs), ld2(U1, i - kFs), ld2(U1, i + kFs), ld2(U1, i + 2 * kFs), C.sdx), m);
    }

    // ---- own pair: strains, products, second derivatives
    const int i = (tx + 2) * kFs + 4 + pz;
    float2 n0, n1, exx, ezz, exz, ezx;   // exz = ux_z, ezx = uz_x
    {
        const float2 am2 = ld2(U0, i - 2 * kFs), am1 = ld2(U0, i - kFs), a00 = ld2(U0, i), ap1 = ld2(U0, i + kFs),
                     ap2 = ld2(U0, i + 2 * kFs);
        const float2 bm2 = ld2(U1, i - 2 * kFs), bm1 = ld2(U1, i - kFs), b00 = ld2(U1, i), bp1 = ld2(U1, i + kFs),
                     bp2 = ld2(U1, i + 2 * kFs);
        const float2 m00 = ld2(MU, i);
        exx = der_x(am2, am1, ap1, ap2, C.sdx);
        ezx = der_x(bm2, bm1, bp1, bp2, C.sdx);
        *reinterpret_cast<float2 *>(S + i) = mul2(ezx, m00);
        const Brk2 bx = brackets2(ld2(MU, i - 2 * kFs), ld2(MU, i - kFs), m00, ld2(MU, i + kFs), ld2(MU, i + 2 * kFs));
        if (VTI) {
            const Brk2 bq = brackets2(ld2(Q, i - 2 * kFs), ld2(Q, i - kFs), ld2(Q, i), ld2(Q, i + kFs), ld2(Q, i + 2 * kFs));
            n0 = mul2(bc2(C.inv_d2x), sum_x(bq, am2, am1, a00, ap1, ap2));
        } else {
            n0 = mul2(bc2(C.inv_d2x), sum_x(twice2(bx), am2, am1, a00, ap1, ap2));
        }
        n1 = mul2(bc2(C.inv_d2x), sum_x(bx, bm2, bm1, b00, bp1, bp2));
    }
    {
        const float2 a00 = ld2(U0, i), alo = ld2(U0, i - 2), ahi = ld2(U0, i + 2);
        const float2 b00 = ld2(U1, i), blo = ld2(U1, i - 2), bhi = ld2(U1, i + 2);
        const float2 m00 = ld2(MU, i), mlo = ld2(MU, i - 2), mhi = ld2(MU, i + 2);
        ezz = der_z(blo, b00, bhi, C.sdz);
        exz = der_z(alo, a00, ahi, C.sdz);
        *reinterpret_cast<float2 *>(R + i) = mul2(exz, m00);
        mixed(i, exx, ezz);
        const Brk2 bz = brackets2(mlo, zsh(mlo, m00), m00, zsh(m00, mhi), mhi);
        n1 = add2(mul2(bc2(C.inv_d2z), sum_z(twice2(bz), blo, b00, bhi)), n1);
        n0 = add2(n0, mul2(bc2(C.inv_d2z), sum_z(bz, alo, a00, ahi)));
    }
    __syncthreads();

    // ---- mixed terms
    auto along_x = [&](const float *p, float s) {
        return der_x(ld2(p, i - 2 * kFs), ld2(p, i - kFs), ld2(p, i + kFs), ld2(p, i + 2 * kFs), s);
    };
    auto along_z = [&](const float *p, float s) { return der_z(ld2(p, i - 2), ld2(p, i), ld2(p, i + 2), s); };
    n0 = add2(n0, along_x(P, VTI ? C.sdx : C.adx));
    n1 = add2(n1, along_z(VTI || AE ? P1 : P, VTI ? C.sdz : C.adz));
    if (AE) {
        n0 = add2(n0, along_x(P1, C.adx));
        n1 = add2(n1, along_z(P, C.adz));
    }
    n1 = add2(n1, along_x(R, C.adx));
    n0 = add2(n0, along_z(S, C.adz));

    const float2 a00 = ld2(U0, i), b00 = ld2(U1, i);
    const int cell = gx * ldz + gz;
    // sources, cell by cell in the reference's order
    if (e0 < e1) {
        const float *srcrow = Sp->src + (long long)it * Sp->nsrc;
        for (int e = e0; e < e1; e++) {
            const InjEntry &E = Sp->inj[e];
            if (E.gx == gx && (E.gz == gz || E.gz == gz + 1)) {
                const float v = E.mt ? (E.wa * srcrow[E.ia] - E.wb * srcrow[E.ib]) : E.wa * srcrow[E.ia];
                if (E.comp == 0) {
                    if (E.gz == gz) n0.x += v;
                    else n0.y += v;
                } else {
                    if (E.gz == gz) n1.x += v;
                    else n1.y += v;
                }
            }
        }
    }
    // receivers (forward): one thread per receiver of this window
    if (!GRAD && (A.flags & F_EXTRACT)) {
        const int r0 = Sp->ext_off[tr.unit], r1 = Sp->ext_off[tr.unit + 1];
        for (int e = r0 + t; e < r1; e += kFt) {
            const ExtEntry &E = Sp->ext[e];
            const float *U = sm + (E.comp == 0 ? L::U0 : L::U1) + (E.gx0 - tr.wx0 + 4) * kFs + (E.gz0 - tr.wz0 + 4);
            float o = 0.f;
#pragma unroll
            for (int a = 0; a < 3; a++)
#pragma unroll
                for (int b = 0; b < 3; b++) o += E.w[a * 3 + b] * U[a * kFs + b];
            Sp->rcv[(long long)it * Sp->nrcv + E.row] = o;
        }
    }
    // leapfrog: dt^2 n / rho + 2 curr - prev, tapered; prev takes its second taper here
    const int oi = tx * kFz + pz;
    float2 p0 = ld2(sm + L::PV0, oi), p1 = ld2(sm + L::PV1, oi);
    const float2 tzx = bc2(txv);
    if (it > 0) {
        p0 = mul2(mul2(p0, tzv), tzx);
        p1 = mul2(mul2(p1, tzv), tzx);
    }
    n0 = mul2(bc2(C.dt2), n0);
    n1 = mul2(bc2(C.dt2), n1);
    div_pairs(n0, n1, ld2(sm + L::RHO, oi), ld2(sm + L::IR, oi));
    const float2 two = bc2(2.f);
    n0 = dif2(fma2(two, a00, n0), p0);   // 2 curr is exact: one rounding
    n1 = dif2(fma2(two, b00, n1), p1);
    n0 = mul2(mul2(n0, tzv), tzx);
    n1 = mul2(mul2(n1, tzv), tzx);
    if (own0 && own1) {
        *reinterpret_cast<float2 *>(pn + cell) = n0;
        *reinterpret_cast<float2 *>(pn + nxz + cell) = n1;
    } else if (own0) {
        pn[cell] = n0.x;
        pn[nxz + cell] = n1.x;
    } else if (own1) {
        pn[cell + 1] = n0.y;
        pn[nxz + cell + 1] = n1.y;
    }
    if (!GRAD && (A.flags & F_STORE) && it % C.sub == 0) {
        const int slot = it / C.sub;
        const long long o = (long long)slot * Sp->snap_slot + cell;
        if (prec == SNAP_FP32 && own0 && own1) {
            *reinterpret_cast<float2 *>((float *)Sp->snap + o) = a00;
            *reinterpret_cast<float2 *>((float *)Sp->snap + o + nxz) = b00;
        } else {
            const float sc = prec == SNAP_FP32 ? 1.f : snap_scale(Sp->snap_amax, slot);
            if (own0) {
                snap_store(Sp->snap, o, prec, a00.x, sc);
                snap_store(Sp->snap, o + nxz, prec, b00.x, sc);
            }
            if (own1) {
                snap_store(Sp->snap, o + 1, prec, a00.y, sc);
                snap_store(Sp->snap, o + nxz + 1, prec, b00.y, sc);
            }
        }
    }

    // ---- zero-lag imaging condition (we_op.cpp:505-562, VTI :1478-1557)
    if (GRAD && do_grad && (own0 || own1)) {
        const float *F0 = sm + L::F0, *F1 = sm + L::F1;
        const float2 t0 = der_x(ld2(F0, i - 2 * kFs), ld2(F0, i - kFs), ld2(F0, i + kFs), ld2(F0, i + 2 * kFs), C.sdx);
        const float2 t2 = der_x(ld2(F1, i - 2 * kFs), ld2(F1, i - kFs), ld2(F1, i + kFs), ld2(F1, i + 2 * kFs), C.sdx);
        const float2 f0 = ld2(F0, i), f1 = ld2(F1, i);
        const float2 t1 = der_z(ld2(F1, i - 2), f1, ld2(F1, i + 2), C.sdz);
        const float2 t3 = der_z(ld2(F0, i - 2), f0, ld2(F0, i + 2), C.sdz);
        float2 dl = make_float2(0.f, 0.f), dm;
        // (two ax0) t0 + ...: doubling is exact, so it commutes with the rounding of every product
        if (!VTI) {
            dm = add2(add2(mul2(add2(exz, ezx), add2(t2, t3)), mul2(mul2(two, exx), t0)), mul2(mul2(two, ezz), t1));
        } else {
            const float2 ev = ld2(sm + L::E, oi), v2 = ld2(sm + L::E + kFo, oi), v3 = ld2(sm + L::E + 2 * kFo, oi);
            const float2 e2 = fma2(two, ev, bc2(1.f));
            const float2 cross = add2(mul2(exx, t1), mul2(ezz, t0));
            dl = add2(add2(mul2(mul2(e2, exx), t0), mul2(ezz, t1)), mul2(v2, cross));
            dm = add2(add2(add2(mul2(add2(exz, ezx), add2(t2, t3)), mul2(mul2(mul2(two, e2), exx), t0)),
                           mul2(mul2(two, ezz), t1)),
                      mul2(v3, cross));
        }
        float2 g0 = ld2(sm + L::G0, oi), g1 = ld2(sm + L::G0 + kFo, oi), g2 = ld2(sm + L::G0 + 2 * kFo, oi);
        const float gw = Sp->gwt[itf];
        const double wdt = (double)gw * 1.0 / (double)A.dtg;
        if (itf > 0) {
            const float2 gd = bc2(gw * A.dtg);
            if (!VTI) g0 = add2(g0, mul2(mul2(gd, add2(exx, ezz)), add2(t0, t1)));
            else g0 = add2(g0, mul2(gd, dl));
            g1 = add2(g1, mul2(gd, dm));
        } else {
            const double wh = (double)gw * 0.5 * (double)A.dtg;
            if (!VTI) {
                const float2 ea = add2(exx, ezz), ta = add2(t0, t1);
                g0.x = (float)((double)g0.x + wh * (double)ea.x * (double)ta.x);
                g0.y = (float)((double)g0.y + wh * (double)ea.y * (double)ta.y);
            } else {
                g0.x = (float)((double)g0.x + wh * (double)dl.x);
                g0.y = (float)((double)g0.y + wh * (double)dl.y);
            }
            g1.x = (float)((double)g1.x + wh * (double)dm.x);
            g1.y = (float)((double)g1.y + wh * (double)dm.y);
        }
        const float2 fp0 = ld2(sm + L::FP0, oi), fp1 = ld2(sm + L::FP0 + kFo, oi);
        const float2 fm0 = ld2(sm + L::FM0, oi), fm1 = ld2(sm + L::FM0 + kFo, oi);
        g2.x = density_term(g2.x, wdt, itf, last, n0.x, n1.x, f0.x, f1.x, fp0.x, fp1.x, fm0.x, fm1.x);
        g2.y = density_term(g2.y, wdt, itf, last, n0.y, n1.y, f0.y, f1.y, fp0.y, fp1.y, fm0.y, fm1.y);
        float *G = Sp->grad + cell;
        if (own0 && own1) {
            *reinterpret_cast<float2 *>(G) = g0;
            *reinterpret_cast<float2 *>(G + nxz) = g1;
            *reinterpret_cast<float2 *>(G + 2 * (long long)nxz) = g2;
        } else if (own0) {
            G[0] = g0.x;
            G[nxz] = g1.x;
            G[2 * (long long)nxz] = g2.x;
        } else {
            G[1] = g0.y;
            G[nxz + 1] = g1.y;
            G[2 * (long long)nxz + 1] = g2.y;
        }
    }
    if (!GRAD && (A.flags & F_AMAX) && (it + 1) % C.sub == 0) {
        float m = 0.f;
        if (own0) m = fmaxf(fabsf(n0.x), fabsf(n1.x));
        if (own1) m = fmaxf(m, fmaxf(fabsf(n0.y), fabsf(n1.y)));
        block_amax(m, sm + L::RED, Sp->snap_amax + (it + 1) / C.sub);
    }
}

// ---------------------------------------------------------------------------
// Band unit: 32 cells along the edge (tangential, lanes) x 6 rows next to it
// (normal, warps 0-5).  XB: left / right edge, normal = x; else top / bottom,
// normal = z.  The arithmetic is the tile kernel's general path through the
// same sbp.cuh routines, except that the coefficient sums of the second
// derivative's closure, which depend on the model only, come ready from
// k_closures: 8 products instead of 8 x 16 operations and a division each.
// ---------------------------------------------------------------------------
template <bool XB, bool VTI, bool GRAD, bool AE>
__device__ __forceinline__ void fused_band(const FusedArgs &A, const ShotDev *__restrict__ Sp, int far, int t0, int own0,
                                           int own1, int unit, int roff, float *sm)
{
    using L = BandLayout<VTI, GRAD>;
    const ModelDev &M = A.M;
    const StepConst &C = A.C;
    const int t = threadIdx.x, it = A.it, lane = t & 31, warp = t >> 5;
    const int nt = Sp->nt, nx = Sp->nx, nz = Sp->nz, ldz = Sp->ldz;
    const int nxz = nx * ldz;
    const int nn = XB ? nx : nz;                       // samples along the normal
    const int nb = far ? nn - kFb : 0;                 // first staged normal sample
    const int prec = C.snap_prec;
    const long long mofs = (long long)Sp->x0 * ldz;
    const int itf = GRAD ? (nt - 1 - (it + 1)) / C.sub : 0;
    const bool do_grad = GRAD && it < nt - 1 && ((nt - 1 - (it + 1)) % C.sub == 0) && (!AE || itf != 0);
    const int last = nt / C.sub;
    constexpr int sx = XB ? kFs : 1, sz = XB ? 1 : kFs;   // shared-memory strides along x and z
    // the unit's tangential range along the grid (z bands: columns clear of the x bands)
    const int tlo = XB ? 0 : 2, thi = XB ? nz : own1 + 4;

    // sample i of a staged array: its shared index, its cell, and whether it exists
    auto sample = [&](int i, int &s, int &o) {
        int c, tt;
        if (XB) { c = i / kFs; tt = i - c * kFs; }
        else { tt = i / kFb; c = i - tt * kFb; }
        const int g = t0 - 4 + tt;
        s = c * kFs + tt;
        o = XB ? (nb + c) * ldz + g : g * ldz + nb + c;
        return g >= tlo && g < thi;
    };
    for (int i = t; i < kFb * kFs; i += kFt) {
        int s, o;
        const bool in = sample(i, s, o);
        sm[L::MU + s] = in ? M.p1[mofs + o] : 0.f;
        sm[L::Q + s] = in ? (VTI ? M.fxx : M.p0)[mofs + o] : 0.f;
        if (VTI) {
            sm[L::LB + s] = in ? M.lbis[mofs + o] : 0.f;
            sm[L::LC + s] = in ? M.c13[mofs + o] : 0.f;
            sm[L::LA + s] = in ? M.p0[mofs + o] : 0.f;
        }
        if (GRAD && do_grad) {
            const long long so = (long long)itf * Sp->snap_slot + o;
            const float inv = prec == SNAP_FP32 ? 1.f : 1.f / snap_scale(Sp->snap_amax, itf);
            sm[L::F0 + s] = in ? snap_load(Sp->snap, so, prec, inv) : 0.f;
            sm[L::F1 + s] = in ? snap_load(Sp->snap, so + nxz, prec, inv) : 0.f;
        }
    }
    // closure coefficients [far][row][sample][tangential] of this unit's cells
    {
        const int ld = XB ? ldz : M.nx, base = (XB ? 0 : Sp->x0) + t0 + lane;
        const bool in = XB ? t0 + lane < nz : t0 + lane < own1;
        for (int k = warp; k < 48; k += kFt / 32) {
            const long long o = (long long)(far * 48 + k) * ld + base;
            sm[L::C0 + k * 32 + lane] = in ? (XB ? Sp->xclos : M.zclos)[o] : 0.f;
            if (VTI && XB) sm[L::C1 + k * 32 + lane] = in ? Sp->xclos[(long long)96 * ldz + o] : 0.f;
        }
    }

    // this thread's cell: normal row k, tangential t0 + lane
    const int k = warp, c = (far ? kFb - 6 : 0) + k, r = far ? 5 - k : k;
    const int gn = nb + c, gt = t0 + lane;
    const int gx = XB ? gn : gt, gz = XB ? gt : gn;
    const bool owned = warp < 6 && gt >= own0 && gt < own1;
    const int cell = gx * ldz + gz;
    const long long mcell = mofs + cell;
    float rho = 1.f, irho = 0.f, tzv = 0.f, txv = 0.f, fp0 = 0.f, fp1 = 0.f, fm0 = 0.f, fm1 = 0.f;
    if (owned) {
        rho = M.p2[mcell];
        irho = M.irho[mcell];
        tzv = Sp->tz[gz];
        txv = Sp->tx[gx];
        if (GRAD && do_grad) {
            if (itf + 1 <= last) {
                const float inv = prec == SNAP_FP32 ? 1.f : 1.f / snap_scale(Sp->snap_amax, itf + 1);
                const long long o = (long long)(itf + 1) * Sp->snap_slot + cell;
                fp0 = snap_load(Sp->snap, o, prec, inv);
                fp1 = snap_load(Sp->snap, o + nxz, prec, inv);
            }
            if (itf > 0) {
                const float inv = prec == SNAP_FP32 ? 1.f : 1.f / snap_scale(Sp->snap_amax, itf - 1);
                const long long o = (long long)(itf - 1) * Sp->snap_slot + cell;
                fm0 = snap_load(Sp->snap, o, prec, inv);
                fm1 = snap_load(Sp->snap, o + nxz, prec, inv);
            }
        }
    }
    const float *curr = Sp->u[(it + 1) & 1];
    float *pn = Sp->u[it & 1];

    pdl_wait();
    pdl_launch();
    if (it >= nt - 1) return;

    for (int i = t; i < kFb * kFs; i += kFt) {
        int s, o;
        const bool in = sample(i, s, o);
        sm[L::U0 + s] = in ? __ldcg(curr + o) : 0.f;
        sm[L::U1 + s] = in ? __ldcg(curr + nxz + o) : 0.f;
    }
    float p0 = 0.f, p1 = 0.f, g0 = 0.f, g1 = 0.f, g2 = 0.f;
    if (owned) {
        p0 = __ldcg(pn + cell);
        p1 = __ldcg(pn + nxz + cell);
        if (GRAD && do_grad) {
            g0 = __ldcg(Sp->grad + cell);
            g1 = __ldcg(Sp->grad + nxz + cell);
            g2 = __ldcg(Sp->grad + 2 * (long long)nxz + cell);
        }
    }
    __syncthreads();

    const float *U0 = sm + L::U0, *U1 = sm + L::U1, *MU = sm + L::MU, *Q = sm + L::Q;
    float *T0 = sm + L::T0, *T1 = sm + L::T1, *CZ = sm + L::CZ, *BX = sm + L::BX;
    // ---- first derivatives on the 8 rows next to the edge, 2 cells beyond the unit along it
    for (int i = t; i < 8 * 36; i += kFt) {
        const int q = i / 36, tt = 2 + i - q * 36, cc = (far ? 2 : 0) + q;
        const int g = t0 - 4 + tt, n = nb + cc;
        // along z a closure reads up to 5 samples from its edge: evaluate where the window holds them
        bool ok = g >= tlo && g < thi;
        if (XB) ok = ok && ((g >= 4 && g < nz - 4) || (g < 4 ? t0 <= 4 : t0 + kFz + 4 >= nz));
        else ok = ok && g >= 4 && g < own1 + 2;
        if (!ok) continue;
        const int s = cc * kFs + tt;
        const int x = XB ? n : g, z = XB ? g : n;
        const float ux_x = d1(U0 + s, sx, x, nx, C.dx, C.sdx);
        const float uz_z = d1(U1 + s, sz, z, nz, C.dz, C.sdz);
        BX[s] = d1(U1 + s, sx, x, nx, C.dx, C.sdx);
        CZ[s] = d1(U0 + s, sz, z, nz, C.dz, C.sdz);
        if (VTI) {
            const float lb = sm[L::LB + s], c13 = sm[L::LC + s], lam = sm[L::LA + s];
            T0[s] = lb * ux_x + c13 * uz_z;
            T1[s] = lam * uz_z + c13 * ux_x;
        } else if (AE) {
            T0[s] = ux_x;
            T1[s] = uz_z;
        } else {
            T0[s] = ux_x + uz_z;
        }
    }
    __syncthreads();

    // receivers of this unit (forward)
    if (!GRAD && (A.flags & F_EXTRACT)) {
        int r0 = 0, r1 = 0, step = 1;
        if (XB) {
            r0 = Sp->ext_off[unit] + t;
            r1 = Sp->ext_off[unit + 1];
            step = kFt;
        } else if (t < own1 - own0) {
            const MarchRow Rr = Sp->mrow[roff + t];
            r0 = Rr.r0;
            r1 = Rr.r1;
        }
        for (int e = r0; e < r1; e += step) {
            const ExtEntry &E = Sp->ext[e];
            const float *U = E.comp == 0 ? U0 : U1;
            const int base = XB ? (E.gx0 - nb) * kFs + E.gz0 - t0 + 4 : (E.gz0 - nb) * kFs + E.gx0 - t0 + 4;
            float o = 0.f;
#pragma unroll
            for (int a = 0; a < 3; a++)
#pragma unroll
                for (int b = 0; b < 3; b++) o += E.w[a * 3 + b] * U[base + a * sx + b * sz];
            Sp->rcv[(long long)it * Sp->nrcv + E.row] = o;
        }
    }

    float amax = 0.f;
    if (owned) {
        const int i = c * kFs + lane + 4;
        const float a00 = U0[i], b00 = U1[i], mu = MU[i];
        // second derivatives: along the normal the closure rows, along the edge the
        // interior form (x bands: the closure again near the corners)
        const float dn2 = XB ? C.d2x : C.d2z, idn2 = XB ? C.inv_d2x : C.inv_d2z;   // inv_d2 is 1/d2 rounded
        const int en = (far ? kFb - 1 : 0) * kFs + lane + 4, dn = far ? -kFs : kFs;
        const float *CL = sm + L::C0 + r * 256 + lane, *CQ = sm + (VTI && XB ? L::C1 : L::C0) + r * 256 + lane;
        float n0 = 0.f, n1 = 0.f;
        if (XB) {
            // ux: x closure of 2 mu (VTI: (1+2eps)2mu), then z with mu; uz: z with 2 mu, then x closure of mu
#pragma unroll
            for (int j = 0; j < 8; j++)
                n0 += div_by((VTI ? CQ[j * 32] : 2.f * CL[j * 32]) * U0[en + j * dn], dn2, idn2);
            if (gz >= 6 && gz < nz - 6) {
                const Brk b = brackets(MU + i, 1);
                n1 = d2i(n1, twice(b), U1 + i, 1, C.inv_d2z);
                n0 = d2i(n0, b, U0 + i, 1, C.inv_d2z);
            } else {
                const bool bot = gz >= 6;
                const int rz = bot ? nz - 1 - gz : gz, d = bot ? -1 : 1;
                const int ez = c * kFs + (bot ? nz - 1 : 0) - t0 + 4;
                const float *zc = M.zclos + (long long)(bot ? 48 : 0) * M.nx + (long long)rz * 8 * M.nx + Sp->x0 + gx;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const float v = zc[(long long)j * M.nx];
                    n1 += div_by((2.f * v) * U1[ez + j * d], C.d2z, C.inv_d2z);
                    n0 += div_by(v * U0[ez + j * d], C.d2z, C.inv_d2z);
                }
            }
#pragma unroll
            for (int j = 0; j < 8; j++) n1 += div_by(CL[j * 32] * U1[en + j * dn], dn2, idn2);
        } else {
            const Brk b = brackets(MU + i, 1);
            if (VTI) n0 = d2i(n0, brackets(Q + i, 1), U0 + i, 1, C.inv_d2x);
            else n0 = d2i(n0, twice(b), U0 + i, 1, C.inv_d2x);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float v = CL[j * 32];
                n1 += div_by((2.f * v) * U1[en + j * dn], dn2, idn2);
                n0 += div_by(v * U0[en + j * dn], dn2, idn2);
            }
            n1 = d2i(n1, b, U1 + i, 1, C.inv_d2x);
        }
        if (AE) {
            n0 += md1(T0 + i, Q + i, sx, gx, nx, C.adx);
            n1 += md1(T1 + i, Q + i, sz, gz, nz, C.adz);
            n0 += md1(T1 + i, Q + i, sx, gx, nx, C.adx);
            n1 += md1(T0 + i, Q + i, sz, gz, nz, C.adz);
        } else if (!VTI) {
            n0 += md1(T0 + i, Q + i, sx, gx, nx, C.adx);
            n1 += md1(T0 + i, Q + i, sz, gz, nz, C.adz);
        } else {
            n0 += d1(T0 + i, sx, gx, nx, C.dx, C.sdx);
            n1 += d1(T1 + i, sz, gz, nz, C.dz, C.sdz);
        }
        n1 += md1(CZ + i, MU + i, sx, gx, nx, C.adx);
        n0 += md1(BX + i, MU + i, sz, gz, nz, C.adz);

        // sources of this cell, in the reference's order
        int e0, e1;
        if (XB) {
            e0 = Sp->inj_off[unit];
            e1 = Sp->inj_off[unit + 1];
        } else {
            const MarchRow Rr = Sp->mrow[roff + gt - own0];
            e0 = Rr.e0;
            e1 = Rr.e1;
        }
        if (e0 < e1) {
            const float *srcrow = Sp->src + (long long)it * Sp->nsrc;
            for (int e = e0; e < e1; e++) {
                const InjEntry &E = Sp->inj[e];
                if (E.gx != gx || E.gz != gz) continue;
                const float v = E.mt ? (E.wa * srcrow[E.ia] - E.wb * srcrow[E.ib]) : E.wa * srcrow[E.ia];
                if (E.comp == 0) n0 += v;
                else n1 += v;
            }
        }
        if (it > 0) {
            p0 = p0 * tzv * txv;
            p1 = p1 * tzv * txv;
        }

        // SAT closures (spatial_operators.hpp:160-822), in the reference's side order
        // (the fluid interface of the acoustic-elastic propagator, its top edge, last)
        const bool edge = gz == 0 || gz == nz - 1 || gx == 0 || gx == nx - 1;
        if (edge) {
            const float lam = VTI ? sm[L::LA + i] : Q[i];
            const float c13 = VTI ? sm[L::LC + i] : lam;
            const float fxx = VTI ? Q[i] : 2 * mu;
            const float lamx = VTI ? sm[L::LB + i] : lam;
            const float imp_s = 0.5f * sqrtf(mu * rho);
            const float imp_p = 0.5f * sqrtf((lam + 2 * mu) * rho);
            const float imp_px = VTI ? 0.5f * sqrtf((1 + 2 * M.eps[mcell]) * (lam + 2 * mu) * rho) : imp_p;
#pragma unroll 1
            for (int q = 0; q < 4; q++) {
                const int side = AE ? (q + 1) & 3 : q;
                const int bc = side == 0 ? C.bc[0] : side == 1 ? C.bc[1] : side == 2 ? C.bc[2] : C.bc[3];
                if (bc != 1 && bc != 2) continue;
                const bool ab = bc == 2;
                if (side < 2) {
                    if (gz != (side == 0 ? 0 : nz - 1)) continue;
                    const int in = side == 0 ? sz : -sz;
                    const float sg = side == 0 ? -1.f : 1.f;
                    float tt = (sg * mu) * tsum(U1 + i, sx, gx, nx) / C.dx + mu * nsum(U0 + i, in) / C.dz;
                    if (ab) tt = tt - imp_s * p0 / C.dt;
                    n0 = n0 - C.sat_z * tt;
                    tt = (sg * c13) * tsum(U0 + i, sx, gx, nx) / C.dx + (2 * mu) * nsum(U1 + i, in) / C.dz;
                    if (ab) tt = tt - imp_p * p1 / C.dt;
                    n1 = n1 - C.sat_z * tt;
                    n1 = n1 - C.nsat_z * lam * ndsum(U1 + i, in);
                } else if (XB) {
                    if (gx != (side == 2 ? 0 : nx - 1)) continue;
                    const int in = side == 2 ? sx : -sx;
                    const float sg = side == 2 ? -1.f : 1.f;
                    float tt = (sg * c13) * tsum(U1 + i, sz, gz, nz) / C.dz + fxx * nsum(U0 + i, in) / C.dx;
                    if (ab) tt = tt - imp_px * p0 / C.dt;
                    n0 = n0 - C.sat_x * tt;
                    n0 = n0 - C.nsat_x * lamx * ndsum(U0 + i, in);
                    tt = (sg * mu) * tsum(U0 + i, sz, gz, nz) / C.dz + mu * nsum(U1 + i, in) / C.dx;
                    if (ab) tt = tt - imp_s * p1 / C.dt;
                    n1 = n1 - C.sat_x * tt;
                }
            }
        }

        n0 = div_by(C.dt2 * n0, rho, irho) + 2 * a00 - p0;
        n1 = div_by(C.dt2 * n1, rho, irho) + 2 * b00 - p1;
        if (edge) {
            const int per = 2 * nx + 2 * nz;
            int kk;
            if (gz == 0) kk = gx;
            else if (gz == nz - 1) kk = nx + gx;
            else if (gx == 0) kk = 2 * nx + gz;
            else kk = 2 * nx + nz + gz;
            n0 = n0 / Sp->den[kk];
            n1 = n1 / Sp->den[per + kk];
        }
        n0 = n0 * tzv * txv;
        if (AE && gz == 0) Sp->halo_save[gx] = p1;   // interface row: coupled and tapered by ae_couple
        else n1 = n1 * tzv * txv;
        pn[cell] = n0;
        pn[nxz + cell] = n1;
        amax = fmaxf(fabsf(n0), fabsf(n1));
        if (!GRAD && (A.flags & F_STORE) && it % C.sub == 0) {
            const int slot = it / C.sub;
            const float sc = prec == SNAP_FP32 ? 1.f : snap_scale(Sp->snap_amax, slot);
            const long long o = (long long)slot * Sp->snap_slot + cell;
            snap_store(Sp->snap, o, prec, a00, sc);
            snap_store(Sp->snap, o + nxz, prec, b00, sc);
        }

        if (GRAD && do_grad) {
            const float *F0 = sm + L::F0, *F1 = sm + L::F1;
            const float ax0 = d1(U0 + i, sx, gx, nx, C.dx, C.sdx), az1 = d1(U1 + i, sz, gz, nz, C.dz, C.sdz);
            const float q0 = d1(F0 + i, sx, gx, nx, C.dx, C.sdx), q1 = d1(F1 + i, sz, gz, nz, C.dz, C.sdz);
            const float q2 = d1(F1 + i, sx, gx, nx, C.dx, C.sdx), q3 = d1(F0 + i, sz, gz, nz, C.dz, C.sdz);
            const float az0 = CZ[i], ax1 = BX[i];
            float dl = 0.f, dm;
            if (!VTI) {
                dm = (az0 + ax1) * (q2 + q3) + 2 * ax0 * q0 + 2 * az1 * q1;
            } else {
                const float e2 = 1 + 2 * M.eps[mcell], v2 = M.gv2[mcell], v3 = M.gv3[mcell];
                dl = e2 * ax0 * q0 + az1 * q1 + v2 * (ax0 * q1 + az1 * q0);
                dm = (az0 + ax1) * (q2 + q3) + 2 * e2 * ax0 * q0 + 2 * az1 * q1 + v3 * (ax0 * q1 + az1 * q0);
            }
            const float gw = Sp->gwt[itf];
            const double wdt = (double)gw * 1.0 / (double)A.dtg;
            if (itf > 0) {
                if (!VTI) g0 = g0 + gw * A.dtg * (ax0 + az1) * (q0 + q1);
                else g0 = g0 + gw * A.dtg * dl;
                g1 = g1 + gw * A.dtg * dm;
            } else {
                const double wh = (double)gw * 0.5 * (double)A.dtg;
                if (!VTI) g0 = (float)((double)g0 + wh * (double)(ax0 + az1) * (double)(q0 + q1));
                else g0 = (float)((double)g0 + wh * (double)dl);
                g1 = (float)((double)g1 + wh * (double)dm);
            }
            float *G = Sp->grad + cell;
            G[0] = g0;
            G[nxz] = g1;
            // interface row: the density term needs the coupled uz (ae_couple)
            if (!AE || gz != 0)
                G[2 * (long long)nxz] = density_term(g2, wdt, itf, last, n0, n1, F0[i], F1[i], fp0, fp1, fm0, fm1);
        }
    }
    if (!GRAD && (A.flags & F_AMAX) && (it + 1) % C.sub == 0)
        block_amax(amax, sm + L::RED, Sp->snap_amax + (it + 1) / C.sub);
}

#ifndef FUSED_FWD_BLOCKS
#define FUSED_FWD_BLOCKS 4
#endif
#ifndef FUSED_GRAD_BLOCKS
#define FUSED_GRAD_BLOCKS 4
#endif
template <bool VTI, bool GRAD, bool AE>
__global__ void __launch_bounds__(kFt, VTI && GRAD ? 3 : (GRAD ? FUSED_GRAD_BLOCKS : FUSED_FWD_BLOCKS))
fused_step(const __grid_constant__ FusedArgs A)
{
    extern __shared__ __align__(16) float sm[];
    const int b = blockIdx.x;
    if (b < A.nxb) {
        const TileRef tr = A.xb[b];
        fused_band<true, VTI, GRAD, AE>(A, A.shots + tr.shot, tr.ox0 != 0, tr.wz0, tr.oz0, tr.oz1, tr.unit, 0, sm);
    } else if (b < A.nxb + A.nzb) {
        const BandRef br = A.zb[b - A.nxb];
        fused_band<false, VTI, GRAD, AE>(A, A.shots + br.shot, br.side, br.xb, br.xb, br.xe, br.unit, br.roff, sm);
    } else {
        fused_interior<VTI, GRAD, AE>(A, A.in[b - A.nxb - A.nzb], sm);
    }
}

// ---------------------------------------------------------------------------
// Closure sums of Dxx_var / Dzz_var (spatial_operators.hpp:31-156): for the
// six rows next to each end of an axis, val[row][j] = sum_k kB2[row][j][k] f[k]
// with the samples counted from that end, in the reference's order.  out:
// [2 ends][6][8][ld], element m of a line at stride `sm`, samples at stride sn.
// ---------------------------------------------------------------------------
__global__ void k_closures(const float *__restrict__ f, float *__restrict__ out, int lines, int ld, int n, long long sl,
                           long long sn)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x, rj = blockIdx.y, far = blockIdx.z;
    if (m >= ld) return;
    const int r = rj >> 3, j = rj & 7;
    float v = 0.f;
    if (m < lines) {
#pragma unroll
        for (int k = 0; k < 8; k++) v += kB2[r][j][k] * f[m * sl + (far ? n - 1 - k : k) * sn];
    }
    out[((long long)far * 48 + rj) * ld + m] = v;
}

void launch_closures(const float *f, float *out, int lines, int ld, int n, long long sl, long long sn, cudaStream_t st)
{
    k_closures<<<dim3((ld + 127) / 128, 48, 2), 128, 0, st>>>(f, out, lines, ld, n, sl, sn);
}

void upload_fused_tables(const float *b1, const float *b2, const float *c2, const float *c1, const float *sc)
{
    cudaMemcpyToSymbol(kB1, b1, sizeof(float) * 24);
    cudaMemcpyToSymbol(kB2, b2, sizeof(float) * 384);
    cudaMemcpyToSymbol(kC2, c2, sizeof(float) * 10);
    cudaMemcpyToSymbol(kC1, c1, sizeof(float) * 2);
    cudaMemcpyToSymbol(kSC, sc, sizeof(float) * 4);
    const float2 one = make_float2(1.f, 1.f), minus = make_float2(-1.f, -1.f);
    cudaMemcpyToSymbol(kOne2, &one, sizeof(one));
    cudaMemcpyToSymbol(kMinus2, &minus, sizeof(minus));
}

template <bool VTI, bool GRAD, bool AE>
static cudaError_t launch_fused_t(const FusedArgs &A, int nin, bool chain, cudaStream_t st)
{
    constexpr size_t bytes = fused_bytes<VTI, GRAD, AE>();
    // a kernel attribute of the current device; cheap, and set before every launch so that no state is shared
    cudaError_t e = cudaFuncSetAttribute(fused_step<VTI, GRAD, AE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(A.nxb + A.nzb + nin);
    cfg.blockDim = dim3(kFt);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = chain ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, fused_step<VTI, GRAD, AE>, A);
}

cudaError_t launch_fused_step(int kind, const ShotDev *shots, const TileRef *xb, int nxb, const BandRef *zb, int nzb,
                              const TileRef *in, int nin, const ModelDev &M, const StepConst &C, int it, int flags,
                              float dtg, bool chain, cudaStream_t st)
{
    if (nxb + nzb + nin <= 0) return cudaSuccess;
    FusedArgs A;
    A.shots = shots;
    A.xb = xb;
    A.zb = zb;
    A.in = in;
    A.nxb = nxb;
    A.nzb = nzb;
    A.M = M;
    A.C = C;
    A.it = it;
    A.flags = flags;
    A.dtg = dtg;
    const bool g = (flags & F_GRAD) != 0;
    if (kind == KIND_VTI)
        return g ? launch_fused_t<true, true, false>(A, nin, chain, st) : launch_fused_t<true, false, false>(A, nin, chain, st);
    if (kind == KIND_AE)
        return g ? launch_fused_t<false, true, true>(A, nin, chain, st) : launch_fused_t<false, false, true>(A, nin, chain, st);
    return g ? launch_fused_t<false, true, false>(A, nin, chain, st) : launch_fused_t<false, false, false>(A, nin, chain, st);
}

}  // namespace fwi2d

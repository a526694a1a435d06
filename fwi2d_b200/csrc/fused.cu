// The whole time loop of a plan in one launch, for elastic, VTI and
// acoustic-elastic grids.
//
// A cooperative launch of resident CTAs (256 threads) advances every shot by
// the steps [it0, it1).  Each CTA keeps the same work units for all of them:
//   x-band     up to 28 z cells of the 6 columns next to the left or right edge;
//   z-band     up to 28 columns of the 6 rows next to the top or bottom edge;
//   interior   a window of 32 (z) x 16 (x) cells clear of the bands.
// Each unit performs the whole step of the reference time loop
// (src/cpp/we_op.cpp:667-871 elastic, :1640-1840 VTI, :2240-2530 the elastic
// grid of the acoustic-elastic propagator) with receivers, snapshots or the
// imaging condition, in the reference's single-precision operation order.
//
// Between steps the CTAs meet at a counter in global memory.  What a launch
// per step costs, and this form does not: B200's SMs start each launch with a
// cold instruction cache (measured on one 81 x 61 shot: about 18 cycles per
// instruction of straight-line code, 12-20 thousand cycles through a band
// unit), the launch gap, and the tail of CTAs.  A CTA stages what no step
// writes (model, closures, snapshots of the imaging condition) before it waits
// for the others, and keeps it in shared memory from step to step when it has
// one unit only.
//
// What bounds it (801 x 401, FP32 snapshots every step, forward / adjoint):
//   one shot     the meetings: 10 of the cycles between a warp's instructions are
//                waits at a barrier; 8.3 / 11.9 us a step, 16.1 / 21.5 in three
//                launches a step;
//   eight shots  latency between a window's halves (0.53 / 0.39 instructions per
//                cycle and scheduler), then the shared-memory pipe (62 / 49 %);
//                47.6 / 81 us a step, 87 / 139 before.
// One 4001 x 1201 shot: 77.6 / 111 us a step, the adjoint at 68 % of a copy's DRAM
// rate (98 B per cell and step).
//
// Everything a step writes is read through L2 (.cg), written by the SM that
// owns the cell and read by its neighbours after the counter.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstring>
#include "engine.h"
#include "sbp.cuh"
#include "snap.cuh"
#include "asat.cuh"
#include "launch.h"

namespace fwi2d {

// (1, 1) and (-1, -1), set at run time: the multipliers of the packed sums (sbp.cuh add2)
static __constant__ float2 kMinus2;

constexpr int kFz = kFusedZ, kFx = kFusedX;      // interior window
constexpr int kFs = kFz + 8;                     // row stride of every staged array (floats)
constexpr int kFt = 256;                         // threads: a z-pair of the interior window each
constexpr int kFu = (kFx + 8) * kFs, kFw = (kFx + 4) * kFs, kFo = kFx * kFz;
constexpr int kFb = 10;                          // band units: samples staged along the normal
constexpr int kBt = kFusedBand + 8;              // and along the edge
static_assert(kFt == kFz / 2 * kFx, "one z-pair per thread");

// 16-byte asynchronous copy through L2; zeros when !ok (nothing is read then)
__device__ __forceinline__ void cp16(float *dst, const float *src, bool ok)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(ok ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ---- tiled bulk copies (TMA) of a window's arrays, issued by one thread -------------
__device__ __forceinline__ unsigned saddr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tma2(float *dst, const CUtensorMap *m, int z, int x, unsigned long long *bar)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                     saddr(dst)),
                 "l"(m), "r"(z), "r"(x), "r"(saddr(bar))
                 : "memory");
}
__device__ __forceinline__ void tma3(float *dst, const CUtensorMap *m, int z, int x, int c, unsigned long long *bar)
{
    asm volatile("cp.async.bulk.tensor.3d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
                     saddr(dst)),
                 "l"(m), "r"(z), "r"(x), "r"(c), "r"(saddr(bar))
                 : "memory");
}
__device__ __forceinline__ void tma4(float *dst, const CUtensorMap *m, int z, int x, int c, int k, unsigned long long *bar)
{
    asm volatile("cp.async.bulk.tensor.4d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
                     saddr(dst)),
                 "l"(m), "r"(z), "r"(x), "r"(c), "r"(k), "r"(saddr(bar))
                 : "memory");
}
__device__ __forceinline__ void bar_init(unsigned long long *bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr(bar)) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned long long *bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_done(unsigned long long *bar, unsigned parity)
{
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok)
                 : "r"(saddr(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}
// Fields and gradients are written by ordinary stores and read by TMA: ordered
// by this fence on the writing side (before the arrival) and on the reading
// side (after the meeting).
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async;" ::: "memory"); }

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

// x / b rounded to nearest single precision from inv, 1/b in double precision
// with a relative error below 2^-51: the quotient of two 24-bit significands
// lies at least 2^-49 (relative) away from every midpoint of two neighbouring
// normal single-precision numbers, so the double product rounds to the same
// number.  No branch, signed zeros included.  A subnormal quotient has fewer bits
// and can be such a midpoint itself: it may then round to the other neighbour,
// 2^-149 away.
__device__ __forceinline__ float div64(float x, double inv) { return (float)((double)x * inv); }

// Both components of a z-pair over the pair's densities b, with r = 1/b rounded
// to single precision: two correction steps of Markstein's division (IBM J.
// Res. Dev. 34, 1990); the first makes the quotient faithful, the second
// rounds it correctly.  Exact while neither the quotient nor the remainder
// leaves the normal range: |x| in [2^-100, 2^100] and b in [2^-20, 2^20]
// (r = 0 marks other b).  Other operands (the field's first, tiny values) take
// the double product.
constexpr float kDivLo = 7.888609052210118e-31f, kDivHi = 1.2676506002282294e30f;
__device__ __forceinline__ double inverse64(float b, float r)
{
    if (!(r > 0.f)) return 1.0 / (double)b;
    // two Newton steps from the 24 good bits of r
    double q = (double)r;
    q = fma(q, fma(-(double)b, q, 1.0), q);
    return fma(q, fma(-(double)b, q, 1.0), q);
}
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
    } else if (!(hi == 0.f && fminf(b.x, b.y) > 0.f)) {
        const double ix = inverse64(b.x, r.x), iy = inverse64(b.y, r.y);
        x0 = make_float2(div64(x0.x, ix), div64(x0.y, iy));
        x1 = make_float2(div64(x1.x, ix), div64(x1.y, iy));
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
constexpr int kWin = 256;   // injection entries of a window that are staged
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
    static constexpr int VAL = E + (VTI && GRAD ? 3 * kFo : 0), KEY = VAL + kWin;   // injected values and their cells
    static constexpr int RED = KEY + kWin;
    static constexpr int FLOATS = RED + 8;
};

// Bands: [10 normal samples, counted from the edge][36 tangential samples] per
// array (row stride kFs), then the closure coefficients of the owned rows,
// [6][8][28], and for x bands those along z next to the corners, [2][6][8][6].
// D, DS, DT: the strain sum (VTI and acoustic-elastic: two arrays) and the two
// shear strains.
constexpr int kVal = 512;
template <bool VTI, bool GRAD, bool AE>
struct BandLayout {
    static constexpr int A = kFb * kFs, CL = 6 * 8 * kFusedBand;
    static constexpr int UN = 0, UT = A, MU = 2 * A, Q = 3 * A, D = 4 * A, DS = 5 * A, DT = 6 * A;
    static constexpr int D1 = 7 * A, LB = D1 + (VTI || AE ? A : 0), LC = LB + (VTI ? A : 0), LA = LC + (VTI ? A : 0);
    static constexpr int F = LA + (VTI ? A : 0);           // snapshots [index & 3][2 components]
    static constexpr int C0 = F + (GRAD ? 8 * A : 0);
    static constexpr int C1 = C0 + CL;                     // VTI x bands: closure of (1+2eps)2mu
    static constexpr int ZC = C1 + (VTI ? CL : 0);
    // per thread, set once per unit: doubles 1/rho and 1/den (two components), then the floats of Slot
    static constexpr int SD = ZC + 2 * 6 * 8 * 6;
    static constexpr int SF = SD + 3 * 2 * kFt;
    static constexpr int SAT = SF + 7 * kFt;               // [own side, corner][along, across, normal][32]
    // injection entries of the unit: up to NVAL of them cached (weights and rows; the forward's moment
    // tensors have two) with this step's values
    static constexpr int NVAL = GRAD ? 512 : 256;
    static constexpr int VAL = SAT + 6 * 32, WA = VAL + NVAL, IA = WA + NVAL, WB = IA + NVAL;
    static constexpr int IB = WB + (GRAD ? 0 : NVAL), VEND = IB + (GRAD ? 0 : NVAL);
    static __device__ __forceinline__ int snap(int k, int c) { return F + ((k & 3) * 2 + c) * A; }
    static constexpr int RED = VEND;
    static constexpr int FLOATS = RED + 8;
    static_assert(SD % 2 == 0, "doubles");
};
constexpr int kCells = 6 * kFusedBand;                     // owned cells of a band unit
// (warps 6 and 7 hold impedances where the others hold their cell's entries)
enum Slot { SL_TZX = 0, SL_TX, SL_IMP, SL_IMPC, SL_R0, SL_R1, SL_NX, SL_E0 = SL_IMP, SL_NZ = SL_IMPC };

template <bool VTI, bool GRAD, bool AE>
constexpr size_t fused_bytes()
{
    return sizeof(float) * (InLayout<VTI, GRAD, AE>::FLOATS > BandLayout<VTI, GRAD, AE>::FLOATS
                                ? InLayout<VTI, GRAD, AE>::FLOATS
                                : BandLayout<VTI, GRAD, AE>::FLOATS);
}

// model arrays of the windows: boxes with the 2-cell halo (mu .. lam), own cells (rho ..)
enum ModelMap { MM_MU = 0, MM_Q, MM_LB, MM_LC, MM_LA, MM_RHO, MM_IR, MM_EPS, MM_V2, MM_V3, MM_COUNT };
struct alignas(64) FusedArgs {
    CUtensorMap mm[MM_COUNT];
    const ShotDev *shots;
    const BandRef *bands;   // x bands (side 2, 3), then z bands (side 0, 1)
    const WinRef *in;
    int nband, nunit;       // band units, all units
    ModelDev M;
    StepConst C;
    int it0, it1, flags;
    float dtg;
    unsigned *count;        // arrivals of this launch's steps, zero at its start
    int *status;            // step + 1 of a wait that gave up
    FluidArgs W;            // acoustic-elastic: the fluid layer
};

// ---- the meeting point of a launch's CTAs -------------------------------------
__device__ __forceinline__ void arrive(unsigned *count)
{
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
}
__device__ __forceinline__ bool reached(const unsigned *count, unsigned target)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
    return v >= target;
}
constexpr int kHardPolls = 1 << 22;
// Waits until every CTA has finished the steps before `it`.  The launch is
// cooperative, so all of them are resident.  Bounded twice: past StepConst::spin
// polls the step is reported, past kHardPolls more the CTA leaves (false), its first
// thread by way of lost_copies().
struct NoCopies {
    __device__ void operator()() const {}
};
template <class Lost = NoCopies>
__device__ __forceinline__ bool meet_at(const unsigned *count, int *status, int spin, unsigned rounds, int it,
                                        Lost lost_copies = Lost())
{
    int lost = 0;
    if (threadIdx.x == 0 && rounds > 0) {
        const unsigned target = rounds * gridDim.x;
        bool ok = false;
        for (int k = 0; k < spin && !ok; k++) ok = reached(count, target);
        if (!ok) {
            atomicCAS(status, 0, it + 1);
            for (int k = 0; k < kHardPolls && !ok; k++) ok = reached(count, target);
            lost = !ok;
            if (lost) lost_copies();
        }
    }
    return !__syncthreads_or(lost);
}
// (acoustic-elastic steps have two meetings: before the step and before its coupling)
template <bool AE, class Lost = NoCopies>
__device__ __forceinline__ bool meet(const FusedArgs &A, int it, Lost lost_copies = Lost())
{
    return meet_at(A.count, A.status, A.C.spin, (AE ? 2u : 1u) * (unsigned)(it - A.it0), it, lost_copies);
}

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

// Waits for a phase of an mbarrier, bounded as `meet`; false when the copies are taken to be lost.
__device__ __forceinline__ bool wait_bar(const FusedArgs &A, unsigned long long *bar, unsigned &parity, int it)
{
    bool ok = false;
    for (int k = 0; k < A.C.spin && !ok; k++) ok = bar_done(bar, parity);
    if (!ok) {
        atomicCAS(A.status, 0, it + 1);
        for (int k = 0; k < kHardPolls && !ok; k++) ok = bar_done(bar, parity);
    }
    parity ^= 1u;
    return ok;
}

// ---------------------------------------------------------------------------
// Interior window.  Thread t owns the z-pair 2 (t & 15) of column t >> 4.  The
// loads come in two groups of tiled bulk copies, issued by one thread: what the
// first half of the work reads (fields with their halo, coefficients: Lead) and
// what the second half reads (previous field, density, snapshots, gradient:
// Own).  While a window is in its second half, the Lead group of the CTA's next
// window is on its way into the arrays that the first half has left, and while
// it is in its first half its own Own group is: a CTA's loads overlap its
// arithmetic without a second buffer.  With a 16-byte cp.async per thread
// instead of the bulk copies, addresses and predicates were 130 of the 420
// instructions per cell (8 forward shots of 801 x 401).
// keep: the model arrays are in shared memory from the last step.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int by(int a, int sub) { return sub == 1 ? a : a / sub; }
struct Imaging {
    int itf, last;
    bool on;
};
template <bool GRAD, bool AE>
__device__ __forceinline__ Imaging imaging(const ShotDev &S, const StepConst &C, int it)
{
    Imaging g = {0, 0, false};
    if (!GRAD) return g;
    const int k = S.nt - 2 - it;
    g.itf = by(k, C.sub);
    g.last = by(S.nt, C.sub);
    g.on = k >= 0 && g.itf * C.sub == k && (!AE || g.itf != 0);
    return g;
}

// by one thread
template <bool VTI, bool GRAD, bool AE>
__device__ __forceinline__ void issue_lead(const FusedArgs &A, const ShotDev &S, const WinRef &tr, int it, bool model,
                                           bool fields, float *sm, unsigned long long *bar)
{
    using L = InLayout<VTI, GRAD, AE>;
    const int z = tr.wz0 - 4, x = tr.wx0 - 2, xm = S.x0 + x;
    if (model) {
        tma2(sm + L::MU, &A.mm[MM_MU], z, xm, bar);
        tma2(sm + L::Q, &A.mm[MM_Q], z, xm, bar);
        if (VTI) {
            tma2(sm + L::LB, &A.mm[MM_LB], z, xm, bar);
            tma2(sm + L::LC, &A.mm[MM_LC], z, xm, bar);
            tma2(sm + L::LA, &A.mm[MM_LA], z, xm, bar);
        }
    }
    if (fields) tma3(sm + L::U0, (const CUtensorMap *)S.maps + SM_LEAD + ((it + 1) & 1), z, x - 2, 0, bar);
}
template <bool VTI>
__device__ __forceinline__ unsigned lead_bytes(bool model)
{
    return 4u * (2 * kFu + (model ? (VTI ? 5 : 2) * kFw : 0));
}

// model: density and its reciprocal (VTI imaging: its coefficients); snapshots (FP32; no step of this launch writes them)
template <bool VTI, bool GRAD, bool AE>
__device__ __forceinline__ void issue_own_static(const FusedArgs &A, const ShotDev &S, const WinRef &tr, int it, bool model,
                                                 float *sm, unsigned long long *bar)
{
    using L = InLayout<VTI, GRAD, AE>;
    const CUtensorMap *sp = (const CUtensorMap *)S.maps;
    const int z = tr.wz0, x = tr.wx0, xm = S.x0 + x;
    const Imaging g = imaging<GRAD, AE>(S, A.C, it);
    const bool snaps = GRAD && g.on, f32 = A.C.snap_prec == SNAP_FP32;
    unsigned bytes = 4u * kFo * (2 + (model ? 2 : 0));
    if (GRAD && g.on) bytes += 4u * kFo * 3;
    if (VTI && GRAD && model) bytes += 4u * kFo * 3;
    const int near = (g.itf + 1 <= g.last ? 2 : 0) + (g.itf > 0 ? 2 : 0);
    if (snaps) bytes += f32 ? 4u * (2 * kFw + kFo * near) : 2u * (2 * kFw + kFx * kFs * near);
    bar_expect(bar, bytes);
    if (model) {
        tma2(sm + L::RHO, &A.mm[MM_RHO], z, xm, bar);
        tma2(sm + L::IR, &A.mm[MM_IR], z, xm, bar);
        if (VTI && GRAD) {
            tma2(sm + L::E, &A.mm[MM_EPS], z, xm, bar);
            tma2(sm + L::E + kFo, &A.mm[MM_V2], z, xm, bar);
            tma2(sm + L::E + 2 * kFo, &A.mm[MM_V3], z, xm, bar);
        }
    }
    if (snaps) {
        const int k = g.itf - S.snap_first, zo = f32 ? z : z - 4;
        tma4(sm + L::F0, sp + SM_SNAP_LEAD, z - 4, x - 2, 0, k, bar);
        if (g.itf + 1 <= g.last) tma4(sm + L::FP0, sp + SM_SNAP_OWN, zo, x, 0, k + 1, bar);
        if (g.itf > 0) tma4(sm + L::FM0, sp + SM_SNAP_OWN, zo, x, 0, k - 1, bar);
        // the next imaging step's new snapshot, from HBM to L2
        if (k >= 2)
            asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global [%0, {%1, %2, %3, %4}];" ::"l"(sp + SM_SNAP_OWN), "r"(zo),
                         "r"(x), "r"(0), "r"(k - 2)
                         : "memory");
    }
}
template <bool VTI, bool GRAD, bool AE>
__device__ __forceinline__ void issue_own_fields(const FusedArgs &A, const ShotDev &S, const WinRef &tr, int it, float *sm,
                                                 unsigned long long *bar)
{
    using L = InLayout<VTI, GRAD, AE>;
    const CUtensorMap *sp = (const CUtensorMap *)S.maps;
    tma3(sm + L::PV0, sp + SM_OWN + (it & 1), tr.wz0, tr.wx0, 0, bar);
    if (GRAD && imaging<GRAD, AE>(S, A.C, it).on) tma3(sm + L::G0, sp + SM_GRAD, tr.wz0, tr.wx0, 0, bar);
}

// Before a CTA leaves a meeting it has given up: the copies of what no step writes that its first
// window has asked for may be on their way into its shared memory.  Both groups also count the
// fields' bytes, which nobody will ask for now; with those taken off, the phases complete once
// the copies have landed.  It works with what is at hand anyway (the phases included): with them
// handed over, or as a call, an adjoint step of 201 x 151 took 8.04 us instead of 7.82.
template <bool GRAD, bool AE>
__device__ __forceinline__ void finish_copies(const FusedArgs &A, const ShotDev &S, int it, unsigned long long *bars)
{
    if (it >= S.nt - 1) return;
    auto landed = [](unsigned long long *bar, unsigned missing) {
        const unsigned phase = bar_done(bar, 0) ? 1 : 0;   // the one that cannot complete yet
        asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(saddr(bar)), "r"(missing) : "memory");
        for (int k = 0; k < kHardPolls && !bar_done(bar, phase); k++) {}
    };
    landed(bars, 4u * 2 * kFu);
    landed(bars + 1, 4u * kFo * (imaging<GRAD, AE>(S, A.C, it).on ? 5 : 2));
}

// 16-bit snapshots of a window lie raw in the F, FP and FM arrays (the own cells' ones in rows
// of kFs, whose first sample keeps the copies' 16-byte alignment); their factors are set by three threads.
__device__ __forceinline__ void set_factors(const ShotDev &S, const Imaging &g, float *inv)
{
    const int d = (int)threadIdx.x - 224;
    if (!g.on || d < 0 || d > 2) return;
    const int k = g.itf - 1 + d;
    if (k >= 0 && k <= g.last) inv[d] = 1.f / snap_scale(S.snap_amax, k);
}
// a pair of raw 16-bit samples at an even index
__device__ __forceinline__ float2 raw2(const float *base, int i, int prec, float inv)
{
    const unsigned w = reinterpret_cast<const unsigned *>(base)[i >> 1];
    float2 v;
    if (prec == SNAP_BF16) v = make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    else v = __half22float2(*reinterpret_cast<const __half2 *>(&w));
    return make_float2(v.x * inv, v.y * inv);
}

// The window's step: wait_lead() before it reads the Lead group, mid() between its halves.
template <bool VTI, bool GRAD, bool AE, bool S16, class Lead, class Mid>
__device__ __forceinline__ bool window_step(const FusedArgs &A, const ShotDev &S, const WinRef &tr, const int it, float *sm,
                                            const float *inv, Lead wait_lead, Mid mid)
{
    using L = InLayout<VTI, GRAD, AE>;
    const StepConst &C = A.C;
    const int t = threadIdx.x, nxz = S.nx * S.ldz, ldz = S.ldz, prec = C.snap_prec;
    const Imaging im = imaging<GRAD, AE>(S, C, it);
    const int itf = im.itf, last = im.last;
    const bool do_grad = im.on;
    const int tx = t >> 4, pz = 2 * (t & 15);
    const int gx = tr.wx0 + tx, gz = tr.wz0 + pz;
    const bool ownx = gx < tr.ox1;
    const bool own0 = ownx && gz >= tr.oz0 && gz < tr.oz1, own1 = ownx && gz + 1 >= tr.oz0 && gz + 1 < tr.oz1;
    float2 tzv = make_float2(0.f, 0.f);   // used in the second half
    float txv = 0.f;
    if (own0 || own1) {
        tzv = *reinterpret_cast<const float2 *>(S.tz + gz);
        txv = S.tx[gx];
    }
    // the window's injected values and their cells and components (entries sorted by cell)
    const int e0 = GRAD ? tr.ea0 : tr.ef0, ne = (GRAD ? tr.ea1 : tr.ef1) - e0;
    const float *srcrow = S.src + (long long)it * S.nsrc;
    if (ne > 0 && ne <= kWin && t < ne) {
        const InjEntry &E = S.inj[e0 + t];
        sm[L::VAL + t] = E.mt ? (E.wa * srcrow[E.ia] - E.wb * srcrow[E.ib]) : E.wa * srcrow[E.ia];
        sm[L::KEY + t] = __int_as_float(2 * ((E.gx - tr.wx0) * kFz + E.gz - tr.wz0) + E.comp);
    }
    const bool here = wait_lead();
    const float *U0 = sm + L::U0 + 2 * kFs, *U1 = sm + L::U1 + 2 * kFs;   // indexed as the 2-halo arrays
    const float *MU = sm + L::MU, *Q = sm + L::Q;
    float *P = sm + L::P, *R = sm + L::R, *T = sm + L::S, *P1 = sm + L::P1;

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
            *reinterpret_cast<float2 *>(T + i) =
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
        *reinterpret_cast<float2 *>(T + i) = mul2(ezx, m00);
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
    // receivers (forward): one thread per receiver of this window
    if (!GRAD && (A.flags & F_EXTRACT)) {
        for (int e = tr.r0 + t; e < tr.r1; e += kFt) {
            const ExtEntry &E = S.ext[e];
            const float *U = sm + (E.comp == 0 ? L::U0 : L::U1) + (E.gx0 - tr.wx0 + 4) * kFs + (E.gz0 - tr.wz0 + 4);
            float o = 0.f;
#pragma unroll
            for (int a = 0; a < 3; a++)
#pragma unroll
                for (int b = 0; b < 3; b++) o += E.w[a * 3 + b] * U[a * kFs + b];
            S.rcv[(long long)it * S.nrcv + E.row] = o;
        }
    }
    const float2 a00 = ld2(U0, i), b00 = ld2(U1, i);
    if (!mid(here)) return false;   // the Own group is there; U and the coefficients are free for the next window

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
    n0 = add2(n0, along_z(T, C.adz));

    const int cell = gx * ldz + gz;
    // sources, cell by cell in the reference's order
    if (ne > 0) {
        auto value = [&](int e) {
            if (ne <= kWin) return sm[L::VAL + e];
            const InjEntry &E = S.inj[e0 + e];
            return E.mt ? (E.wa * srcrow[E.ia] - E.wb * srcrow[E.ib]) : E.wa * srcrow[E.ia];
        };
        auto key = [&](int e) {
            if (ne <= kWin) return __float_as_int(sm[L::KEY + e]);
            const InjEntry &E = S.inj[e0 + e];
            return 2 * ((E.gx - tr.wx0) * kFz + E.gz - tr.wz0) + E.comp;
        };
        const int k = 2 * (tx * kFz + pz);   // of the pair's first cell: keys k .. k + 3
        int lo = 0, hi = ne;
        while (lo < hi) {
            const int m = (lo + hi) >> 1;
            if (key(m) < k) lo = m + 1;
            else hi = m;
        }
        for (; lo < ne && key(lo) <= k + 3; lo++) {
            const float v = value(lo);
            const int d = key(lo) - k;
            if (d == 0) n0.x += v;
            else if (d == 1) n1.x += v;
            else if (d == 2) n0.y += v;
            else n1.y += v;
        }
    }
    float *pn = S.u[it & 1];   // prev in, next out
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
    const int slot = by(it, C.sub);
    if (!GRAD && (A.flags & F_STORE) && slot * C.sub == it) {
        const long long o = (long long)slot * S.snap_slot + cell;
        if (prec == SNAP_FP32 && own0 && own1) {
            *reinterpret_cast<float2 *>((float *)S.snap + o) = a00;
            *reinterpret_cast<float2 *>((float *)S.snap + o + nxz) = b00;
        } else {
            const float sc = prec == SNAP_FP32 ? 1.f : snap_scale(S.snap_amax, slot);
            if (own0) {
                snap_store(S.snap, o, prec, a00.x, sc);
                snap_store(S.snap, o + nxz, prec, b00.x, sc);
            }
            if (own1) {
                snap_store(S.snap, o + 1, prec, a00.y, sc);
                snap_store(S.snap, o + nxz + 1, prec, b00.y, sc);
            }
        }
    }

    // ---- zero-lag imaging condition (we_op.cpp:505-562, VTI :1478-1557)
    if (GRAD && do_grad && (own0 || own1)) {
        auto f = [&](int c, int j) {
            if (S16) return raw2(sm + L::F0, c * kFw + j, prec, inv[1]);
            return ld2(sm + L::F0, c * kFw + j);
        };
        const float2 t0 = der_x(f(0, i - 2 * kFs), f(0, i - kFs), f(0, i + kFs), f(0, i + 2 * kFs), C.sdx);
        const float2 t2 = der_x(f(1, i - 2 * kFs), f(1, i - kFs), f(1, i + kFs), f(1, i + 2 * kFs), C.sdx);
        const float2 f0 = f(0, i), f1 = f(1, i);
        const float2 t1 = der_z(f(1, i - 2), f1, f(1, i + 2), C.sdz);
        const float2 t3 = der_z(f(0, i - 2), f0, f(0, i + 2), C.sdz);
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
        const float gw = S.gwt[itf];
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
        auto near = [&](int base, int c, float iv) {
            if (S16) return raw2(sm + base, c * kFx * kFs + tx * kFs + pz + 4, prec, iv);
            return ld2(sm + base + c * kFo, oi);
        };
        const float iv0 = S16 ? inv[0] : 1.f, iv2 = S16 ? inv[2] : 1.f;
        // no snapshot follows the last one, which is also the first where sub exceeds the record: nothing is
        // loaded for it then, and it counts as zero
        const bool next = itf + 1 <= last;
        const float2 none = make_float2(0.f, 0.f);
        const float2 fp0 = next ? near(L::FP0, 0, iv2) : none, fp1 = next ? near(L::FP0, 1, iv2) : none;
        const float2 fm0 = near(L::FM0, 0, iv0), fm1 = near(L::FM0, 1, iv0);
        g2.x = density_term(g2.x, wdt, itf, last, n0.x, n1.x, f0.x, f1.x, fp0.x, fp1.x, fm0.x, fm1.x);
        g2.y = density_term(g2.y, wdt, itf, last, n0.y, n1.y, f0.y, f1.y, fp0.y, fp1.y, fm0.y, fm1.y);
        float *G = S.grad + cell;
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
        block_amax(m, sm + L::RED, S.snap_amax + (it + 1) / C.sub);
    }
    return true;
}

// ---------------------------------------------------------------------------
// Band unit: up to 28 cells along the edge (tangential, lanes 2-29) x 6 rows
// next to it (warps 0-5).  XB: left / right edge, the normal is x; else top /
// bottom, the normal is z.  In the components and axes along (t) and across
// (n) the edge the operators of all four sides are the same; samples along the
// normal are counted from the edge, which turns the sign (sg) of the far
// side's first normal derivatives and leaves every rounding as it was
// (s -= B b is s += (-B) b).  A row is uniform across a warp, so that the
// closures' rows do not diverge.  The coefficient sums of the second
// derivative's closure depend on the model only and come ready from
// k_closures: 8 products and quotients instead of 8 x 16 operations.
// One such CTA sets the time of a step on small plans, and its time is one
// warp's chain of instructions: so the SAT terms of the edge row, which need
// the fields only, are formed by warps 6 and 7 beside the rows' derivatives,
// and whatever depends on the model alone is set up once per unit (keep).  In
// the adjoint such a CTA holds the three snapshots around the imaging time and
// fetches the next one a step ahead (one: the CTA has this unit only; ring: the
// snapshots are there from the last step).
// ---------------------------------------------------------------------------
template <bool XB, bool VTI, bool GRAD, bool AE>
__device__ __forceinline__ bool fused_band(const FusedArgs &A, const BandRef br, const int it, const bool first,
                                           const bool keep, const bool one, bool &ring, float *sm)
{
    using L = BandLayout<VTI, GRAD, AE>;
    const ModelDev &M = A.M;
    const StepConst &C = A.C;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const ShotDev *__restrict__ Sp = A.shots + br.shot;
    const int nt = Sp->nt, nx = Sp->nx, nz = Sp->nz, ldz = Sp->ldz;
    const int nxz = nx * ldz;
    const bool far = br.side & 1;
    const int t0 = br.xb, t1 = br.xe;                  // owned cells along the edge
    const int nn = XB ? nx : nz;
    const int prec = C.snap_prec;
    const long long mofs = (long long)Sp->x0 * ldz;
    const Imaging im = imaging<GRAD, AE>(*Sp, C, it);
    const int itf = im.itf, last = im.last;
    const bool do_grad = im.on;
    const float sg = far ? -1.f : 1.f;
    // along the edge: samples that exist (z bands: within the columns clear of the x bands and their halo)
    const int glo = XB ? 0 : t0 - 4, ghi = XB ? nz : t1 + 4;

    // the two staged samples of this thread: shared index, cell, and whether they exist
    int s_[2], o_[2];
    bool in_[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int i = t + h * kFt;
        int c, tt;
        if (XB) { c = i / kBt; tt = i - c * kBt; }
        else { tt = i / kFb; c = i - tt * kFb; }
        const int g = t0 - 4 + tt, gn = far ? nn - 1 - c : c;
        const bool slot = i < kFb * kBt;
        in_[h] = slot && g >= glo && g < ghi;
        s_[h] = slot ? c * kFs + tt : -1;
        o_[h] = in_[h] ? (XB ? gn * ldz + g : g * ldz + gn) : 0;
    }
    static_assert(kFb * kBt <= 2 * kFt, "two samples per thread");
    auto stage = [&](int dst, const float *src) {
#pragma unroll
        for (int h = 0; h < 2; h++)
            if (s_[h] >= 0) sm[dst + s_[h]] = in_[h] ? src[o_[h]] : 0.f;
    };

    // this thread's cell: row `warp` from the edge, tangential t0 + lane - 2; warps 6
    // and 7 take the edge row (its SAT terms along and across the edge)
    const int row = warp < 6 ? warp : 0;
    const int gt = t0 + lane - 2, gn = far ? nn - 1 - row : row;
    const int gx = XB ? gn : gt, gz = XB ? gt : gn;
    const bool mine = lane >= 2 && gt < t1, owned = mine && warp < 6;
    const int cell = mine ? gx * ldz + gz : 0;
    const long long mcell = mofs + cell;
    // x bands: the corner cells' rows along the top or bottom edge, one per lane of warps 6 and 7
    const bool top_here = XB && t0 == 0, bot_here = XB && t1 == nz;
    const bool cside = warp >= 6 && lane < 6 && (top_here || bot_here);
    const int cgx = far ? nx - 1 - lane : lane, cgz = top_here ? 0 : nz - 1;
    const int ccell = cside ? cgx * ldz + cgz : 0;
    double *SD = reinterpret_cast<double *>(sm + L::SD) + t;
    float *SF = sm + L::SF + t;

    if (!keep) {
        stage(L::MU, M.p1 + mofs);
        stage(L::Q, (VTI ? M.fxx : M.p0) + mofs);
        if (VTI) {
            stage(L::LB, M.lbis + mofs);
            stage(L::LC, M.c13 + mofs);
            stage(L::LA, M.p0 + mofs);
        }
        // closure coefficients [row][sample][tangential] of the owned cells
        const int ld = XB ? ldz : M.nx, base = (XB ? 0 : Sp->x0) + t0;
        for (int i = t; i < L::CL; i += kFt) {
            const int k = i / kFusedBand, q = i - k * kFusedBand;
            const bool in = t0 + q < t1;
            const long long o = (long long)((far ? 48 : 0) + k) * ld + base + q;
            sm[L::C0 + i] = in ? (XB ? Sp->xclos : M.zclos)[o] : 0.f;
            if (VTI && XB) sm[L::C1 + i] = in ? Sp->xclos[(long long)96 * ldz + o] : 0.f;
        }
        if (XB)   // along z next to the corners: [top, bottom][row][sample][column]
            for (int i = t; i < 2 * 48 * 6; i += kFt) {
                const int k = i / 6, c = i - 6 * k;
                sm[L::ZC + i] = M.zclos[(long long)k * M.nx + Sp->x0 + (far ? nx - 1 - c : c)];
            }
        // impedance of a side's SAT at model cell m: warp 6 the shear one, warp 7 the compressional one
        auto impedance = [&](long long m, bool zside) {
            const float mu = M.p1[m], rho = M.p2[m];
            if (warp == 6) return 0.5f * sqrtf(mu * rho);
            const float l2m = M.p0[m] + 2 * mu;
            return VTI && !zside ? 0.5f * sqrtf((1 + 2 * M.eps[m]) * l2m * rho) : 0.5f * sqrtf(l2m * rho);
        };
        float tzv = 0.f, txv = 0.f;
        int4 ent = make_int4(0, 0, 0, 0);
        int r0 = 0, r1 = 0;
        if (mine) {
            SD[0] = 1.0 / (double)M.p2[mcell];
            if (warp >= 6) SF[SL_IMP * kFt] = impedance(mcell, !XB);
            if (gz == 0 || gz == nz - 1 || gx == 0 || gx == nx - 1) {
                const int per = 2 * nx + 2 * nz;
                const int kk = gz == 0 ? gx : gz == nz - 1 ? nx + gx : gx == 0 ? 2 * nx + gz : 2 * nx + nz + gz;
                SD[kFt] = 1.0 / (double)Sp->den[kk];
                SD[2 * kFt] = 1.0 / (double)Sp->den[per + kk];
            }
            tzv = Sp->tz[gz];
            txv = Sp->tx[gx];
            if (owned) ent = Sp->brange[(long long)br.unit * kCells + row * kFusedBand + lane - 2];
            if (!XB) {
                const MarchRow R = Sp->mrow[br.roff + gt - t0];
                r0 = R.r0;
                r1 = warp == 0 ? R.r1 : R.r0;
            }
        }
        if (XB) {
            r0 = Sp->ext_off[br.unit] + t;
            r1 = Sp->ext_off[br.unit + 1];
        }
        if (cside) SF[SL_IMPC * kFt] = impedance(mofs + ccell, true);
        SF[SL_TZX * kFt] = tzv;
        SF[SL_TX * kFt] = txv;
        if (warp < 6) {
            SF[SL_E0 * kFt] = __int_as_float(ent.x);
            SF[SL_NX * kFt] = __int_as_float(ent.y);
            SF[SL_NZ * kFt] = __int_as_float(ent.z);
        }
        SF[SL_R0 * kFt] = __int_as_float(r0);
        SF[SL_R1 * kFt] = __int_as_float(r1);
    }
    // loads that nothing waits for yet: the rows of this step's injected values, the snapshot two
    // imaging times on; then the snapshots around this one where they are not there from the last step
    const int inj0 = Sp->inj_off[br.unit], ninj = Sp->inj_off[br.unit + 1] - inj0;
    const bool cached = ninj <= L::NVAL, act = it < nt - 1;
    const float *srcrow = Sp->src + (long long)it * Sp->nsrc;
    constexpr int NE = L::NVAL / kFt;
    if (!one && act && cached) {
        for (int e = t; e < ninj; e += kFt) {
            const InjEntry &E = Sp->inj[inj0 + e];
            sm[L::VAL + e] = E.mt ? (E.wa * srcrow[E.ia] - E.wb * srcrow[E.ib]) : E.wa * srcrow[E.ia];
        }
    }
    if (one && !keep && cached) {
#pragma unroll
        for (int h = 0; h < NE; h++) {
            const int e = t + h * kFt;
            if (e < ninj) {
                const InjEntry E = Sp->inj[inj0 + e];
                sm[L::WA + e] = E.wa;
                sm[L::IA + e] = __int_as_float(E.ia);
                if (!GRAD) {
                    sm[L::WB + e] = E.wb;
                    sm[L::IB + e] = __int_as_float(E.mt ? E.ib : -1);
                }
            }
        }
    }
    float sv[NE], sw = 0.f;
#pragma unroll
    for (int h = 0; h < NE; h++) {
        const int e = t + h * kFt;
        sv[h] = 0.f;
        if (one && act && cached && e < ninj) {
            const int ia = __float_as_int(sm[L::IA + e]);
            sv[h] = srcrow[ia];
            if (!GRAD) {
                const int ib = __float_as_int(sm[L::IB + e]);
                if (ib >= 0) sw = srcrow[ib];
            }
            asm volatile("prefetch.global.L2 [%0];" ::"l"(srcrow + Sp->nsrc + ia));
        }
    }
    float na_[2] = {0.f, 0.f}, nb_[2] = {0.f, 0.f};
    const bool more = GRAD && do_grad && itf - Sp->snap_first >= 2;
    if (GRAD && do_grad) {
        auto load = [&](int k, float (&a)[2], float (&b)[2]) {
            const float inv = prec == SNAP_FP32 ? 1.f : 1.f / snap_scale(Sp->snap_amax, k);
            const long long so = (long long)k * Sp->snap_slot;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                a[h] = in_[h] ? snap_load(Sp->snap, so + o_[h], prec, inv) : 0.f;
                b[h] = in_[h] ? snap_load(Sp->snap, so + o_[h] + nxz, prec, inv) : 0.f;
            }
        };
        if (ring) {
            if (more) load(itf - 2, na_, nb_);
        } else {
            // the window at this time; the neighbours at the own cells (a unit that is kept: their windows)
            float a[2], b[2];
            auto own = [&](int k, bool have, float &x, float &y) {
                x = y = 0.f;
                if (!owned || !have) return;
                const float inv = prec == SNAP_FP32 ? 1.f : 1.f / snap_scale(Sp->snap_amax, k);
                x = snap_load(Sp->snap, (long long)k * Sp->snap_slot + cell, prec, inv);
                y = snap_load(Sp->snap, (long long)k * Sp->snap_slot + cell + nxz, prec, inv);
            };
            auto put = [&](int k) {
#pragma unroll
                for (int h = 0; h < 2; h++)
                    if (s_[h] >= 0) {
                        sm[L::snap(k, 0) + s_[h]] = a[h];
                        sm[L::snap(k, 1) + s_[h]] = b[h];
                    }
            };
            float fp0, fp1, fm0, fm1;
            load(itf, a, b);
            own(itf + 1, itf + 1 <= last, fp0, fp1);
            own(itf - 1, !one && itf > 0, fm0, fm1);
            put(itf);
            const int c = row * kFs + lane + 2;
            if (owned) {
                sm[L::snap(itf + 1, 0) + c] = fp0;
                sm[L::snap(itf + 1, 1) + c] = fp1;
            }
            if (one) {
                if (itf > 0) {
                    load(itf - 1, a, b);
                    put(itf - 1);
                }
                if (more) load(itf - 2, na_, nb_);
            } else if (owned) {
                sm[L::snap(itf - 1, 0) + c] = fm0;
                sm[L::snap(itf - 1, 1) + c] = fm1;
            }
        }
        ring = one;
    }
    const bool edge = owned && (gz == 0 || gz == nz - 1 || gx == 0 || gx == nx - 1);
    const float *curr = Sp->u[(it + 1) & 1];
    float *pn = Sp->u[it & 1];

    if (first && !meet<AE>(A, it)) return false;
    if (it >= nt - 1) return true;

    float p0 = 0.f, p1 = 0.f, g0 = 0.f, g1 = 0.f, g2 = 0.f, c0 = 0.f, c1 = 0.f;
    {
        float a_[2], b_[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            a_[h] = in_[h] ? __ldcg(curr + o_[h] + (XB ? 0 : nxz)) : 0.f;
            b_[h] = in_[h] ? __ldcg(curr + o_[h] + (XB ? nxz : 0)) : 0.f;
        }
        if (mine) {
            p0 = __ldcg(pn + cell);
            p1 = __ldcg(pn + nxz + cell);
        }
        if (cside) {
            c0 = __ldcg(pn + ccell);
            c1 = __ldcg(pn + nxz + ccell);
        }
        if (GRAD && do_grad && owned) {
            g0 = __ldcg(Sp->grad + cell);
            g1 = __ldcg(Sp->grad + nxz + cell);
            g2 = __ldcg(Sp->grad + 2 * (long long)nxz + cell);
        }
#pragma unroll
        for (int h = 0; h < 2; h++)
            if (s_[h] >= 0) {
                sm[L::UN + s_[h]] = a_[h];
                sm[L::UT + s_[h]] = b_[h];
                if (GRAD && more && one) {
                    sm[L::snap(itf - 2, 0) + s_[h]] = na_[h];
                    sm[L::snap(itf - 2, 1) + s_[h]] = nb_[h];
                }
            }
#pragma unroll
        for (int h = 0; h < NE; h++) {
            const int e = t + h * kFt;
            if (one && cached && e < ninj) {
                float v = sm[L::WA + e] * sv[h];
                if (!GRAD && __float_as_int(sm[L::IB + e]) >= 0) v = v - sm[L::WB + e] * sw;
                sm[L::VAL + e] = v;
            }
        }
    }
    __syncthreads();

    const float ssn = XB ? C.sdx : C.sdz, sst = XB ? C.sdz : C.sdx, adn = XB ? C.adx : C.adz, adt = XB ? C.adz : C.adx;
    const double idn = XB ? C.idx64 : C.idz64, idt = XB ? C.idz64 : C.idx64;
    const double idn2 = XB ? C.id2x64 : C.id2z64;
    const float inv_d2t = XB ? C.inv_d2z : C.inv_d2x;
    const int i = warp * kFs + lane + 2;      // this thread's sample
    // x bands: z closures along the edge; zo / zs: the end's sample relative to this one and the way in
    const int zr = XB ? (gz < nz - 1 - gz ? gz : nz - 1 - gz) : 6;
    const bool zfar = XB && gz >= nz - 1 - gz;
    const int zo = XB ? (zfar ? nz - 1 - gz : -gz) : 0, zs = zfar ? -1 : 1;

    // first derivatives at sample i of array p (row `warp`)
    auto dern = [&](int p) {
        const float *u = sm + p + i;
        if (warp >= 4)
            return sg * (ssn * (kC1[0] * (u[kFs] - u[-kFs]) + kC1[1] * (u[2 * kFs] - u[-2 * kFs])));
        const float *b = sm + p + lane + 2;
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 6; k++) s += kB1[warp][k] * b[k * kFs];
        return div64(sg * s, idn);
    };
    // sum of the closure row along the edge (x bands near the corners), without the division
    auto zsum = [&](const float *u) {
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 6; k++) s += ((zfar ? -1.f : 1.f) * kB1[zr][k]) * u[zo + k * zs];
        return s;
    };
    auto dert = [&](int p) {
        const float *u = sm + p + i;
        if (XB && zr < 4) return div64(zsum(u), idt);
        return sst * (kC1[0] * (u[1] - u[-1]) + kC1[1] * (u[2] - u[-2]));
    };
    // first derivatives of products of arrays p and q
    auto mdern = [&](int p, int q) {
        const float *u = sm + p + i, *v = sm + q + i;
        if (warp >= 4)
            return sg * (adn * (kC1[0] * (u[kFs] * v[kFs] - u[-kFs] * v[-kFs]) +
                                kC1[1] * (u[2 * kFs] * v[2 * kFs] - u[-2 * kFs] * v[-2 * kFs])));
        const float *b = sm + p + lane + 2, *c = sm + q + lane + 2;
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 6; k++) s += kB1[warp][k] * b[k * kFs] * c[k * kFs];
        return adn * (sg * s);
    };
    auto mdert = [&](int p, int q) {
        const float *u = sm + p + i, *v = sm + q + i;
        if (XB && zr < 4) {
            float s = 0.f;
#pragma unroll
            for (int k = 0; k < 6; k++)
                s += ((zfar ? -1.f : 1.f) * kB1[zr][k]) * u[zo + k * zs] * v[zo + k * zs];
            return adt * s;
        }
        return adt * (kC1[0] * (u[1] * v[1] - u[-1] * v[-1]) + kC1[1] * (u[2] * v[2] - u[-2] * v[-2]));
    };

    // ---- first derivatives on the 8 rows next to the edge, 2 cells beyond the unit along it.
    // Near a corner the closure's samples have to lie in the staged window: other points are never used.
    float en = 0.f, et = 0.f, es = 0.f, eq = 0.f;   // d_n un, d_t ut, d_n ut, d_t un
    if (gt >= glo && gt < ghi) {
        en = dern(L::UN);
        es = dern(L::UT);
        if (!XB || zr >= 4 || (zfar ? nz - 1 - t0 + 4 < kBt : t0 - 4 <= 0)) {
            et = dert(L::UT);
            eq = dert(L::UN);
        }
        if (VTI) {
            const float lb = sm[L::LB + i], lc = sm[L::LC + i], la = sm[L::LA + i];
            sm[L::D + i] = (XB ? lb : la) * en + lc * et;
            sm[L::D1 + i] = (XB ? la : lb) * et + lc * en;
        } else if (AE) {
            sm[L::D + i] = en;
            sm[L::D1 + i] = et;
        } else {
            sm[L::D + i] = en + et;
        }
        sm[L::DS + i] = es;
        sm[L::DT + i] = eq;
    }
    __syncthreads();

    // receivers of this unit (forward)
    if (!GRAD && (A.flags & F_EXTRACT)) {
        const int r1 = __float_as_int(SF[SL_R1 * kFt]);
        for (int e = __float_as_int(SF[SL_R0 * kFt]); e < r1; e += XB ? kFt : 1) {
            const ExtEntry &E = Sp->ext[e];
            const bool nc = XB ? E.comp == 0 : E.comp == 1;
            const int gn0 = XB ? E.gx0 : E.gz0, gt0 = XB ? E.gz0 : E.gx0;
            const float *U = sm + (nc ? L::UN : L::UT) + (far ? nn - 1 - gn0 : gn0) * kFs + gt0 - t0 + 4;
            const int sn = far ? -kFs : kFs;
            float o = 0.f;
#pragma unroll
            for (int a = 0; a < 3; a++)
#pragma unroll
                for (int b = 0; b < 3; b++) o += E.w[a * 3 + b] * U[XB ? a * sn + b : b * sn + a];
            Sp->rcv[(long long)it * Sp->nrcv + E.row] = o;
        }
    }

    const float tzv = SF[SL_TZX * kFt], txv = SF[SL_TX * kFt];
    if (it > 0) {
        p0 = p0 * tzv * txv;
        p1 = p1 * tzv * txv;
    }
    float pn_ = XB ? p0 : p1, pt_ = XB ? p1 : p0;   // previous values
    if (warp >= 6) {
        // SAT terms (spatial_operators.hpp:160-822) of one side at one cell, scaled as they are subtracted:
        // warp 6 the term of the component along the side, warp 7 that of the component across it and its
        // normal-derivative term.  v: the component across, w: along; at: the cell's sample; row k of the band;
        // own: the side is the band's edge, else the top or bottom edge at a corner.
        auto sat_terms = [&](bool own, int side, int at, int k, float prev, float imp, float *out) {
            const int bc = side == 0 ? C.bc[0] : side == 1 ? C.bc[1] : side == 2 ? C.bc[2] : C.bc[3];
            const bool zside = side < 2, ab = bc == 2;
            const float *v = sm + (own ? L::UN : L::UT) + at, *w = sm + (own ? L::UT : L::UN) + at;
            const float *q = warp == 6 ? v : w;   // the derivative along the side is that of the other component
            const int in = own ? kFs : (side & 1 ? -1 : 1);
            const double ia = own ? idt : idn, ic = own ? idn : idt;
            const float mu = sm[L::MU + at], lam = VTI ? sm[L::LA + at] : sm[L::Q + at];
            float s = 0.f;
            if (own) {
                const int g = XB ? t0 - 4 + at : 6;   // position along z (edge row: `at` is the tangential sample)
                if (XB && (g < 4 || g >= nz - 4)) {
                    const bool f = g >= 4;
                    const int r = f ? nz - 1 - g : g, o = f ? r : -r, d = f ? -1 : 1;
                    const float e = f ? -1.f : 1.f;
#pragma unroll
                    for (int j = 0; j < 6; j++) s += (e * kB1[r][j]) * q[o + j * d];
                } else {
                    s += kC1[0] * (q[1] - q[-1]);
                    s += kC1[1] * (q[2] - q[-2]);
                }
            } else {
                if (k >= 4) {
                    s += kC1[0] * (q[kFs] - q[-kFs]);
                    s += kC1[1] * (q[2 * kFs] - q[-2 * kFs]);
                } else {
#pragma unroll
                    for (int j = 0; j < 6; j++) s += kB1[k][j] * q[(j - k) * kFs];
                }
                s = sg * s;
            }
            const float s2 = side & 1 ? 1.f : -1.f, sat = zside ? C.sat_z : C.sat_x;
            const float *u = warp == 6 ? w : v;   // the component itself: one-sided derivative into the domain
            float nv = 0.f, nd = 0.f;
#pragma unroll
            for (int j = 0; j < 4; j++) nv += kSC[j] * u[j * in];
#pragma unroll
            for (int j = 0; j < 6; j++) nd -= kB1[0][j] * u[j * in];
            const float c13 = VTI ? sm[L::LC + at] : lam, fxx = VTI ? sm[L::Q + at] : 2 * mu;
            const float ca = warp == 6 ? mu : c13, cn = warp == 6 ? mu : (zside ? 2 * mu : fxx);
            float tt = div64((s2 * ca) * s, ia) + div64(cn * nv, ic);
            if (ab) tt = tt - div64(imp * prev, C.idt64);
            if (warp == 6) {
                out[0] = sat * tt;
            } else {
                out[32] = sat * tt;
                out[64] = (zside ? C.nsat_z : C.nsat_x) * (zside || !VTI ? lam : sm[L::LB + at]) * nd;
            }
        };
        if (mine) {
            const int bc = br.side == 0 ? C.bc[0] : br.side == 1 ? C.bc[1] : br.side == 2 ? C.bc[2] : C.bc[3];
            if (bc == 1 || bc == 2)
                sat_terms(true, br.side, lane + 2, 0, warp == 6 ? pt_ : pn_, SF[SL_IMP * kFt], sm + L::SAT + lane);
        }
        if (cside) {
            const float ctz = Sp->tz[cgz], ctx = Sp->tx[cgx];
            float c = warp == 6 ? c0 : c1;   // along the top or bottom edge: ux, across: uz
            if (it > 0) c = c * ctz * ctx;
            const int bc = top_here ? C.bc[0] : C.bc[1];
            if (bc == 1 || bc == 2)
                sat_terms(false, top_here ? 0 : 1, lane * kFs + cgz - t0 + 4, lane, c, SF[SL_IMPC * kFt],
                          sm + L::SAT + 96 + lane);
        }
    }

    float amax = 0.f, an = 0.f, at = 0.f, un = 0.f, ut = 0.f;
    if (owned) {
        un = sm[L::UN + i];
        ut = sm[L::UT + i];
        // second derivatives: the closure rows across the edge, the interior form along it
        // (x bands: the closure again near the corners); acc += val u / d^2, sample by sample
        const float *CL = sm + L::C0 + warp * 8 * kFusedBand + lane - 2;
        const float *CQ = sm + (VTI && XB ? L::C1 : L::C0) + warp * 8 * kFusedBand + lane - 2;
        const float *UN = sm + L::UN + lane + 2, *UT = sm + L::UT + lane + 2;
#pragma unroll
        for (int j = 0; j < 8; j++)
            an += div64((VTI && XB ? CQ[j * kFusedBand] : 2.f * CL[j * kFusedBand]) * UN[j * kFs], idn2);
        if (XB && zr < 6) {
            const float *zc = sm + L::ZC + (zfar ? 288 : 0) + zr * 48 + warp;
            const float *vn = sm + L::UN + i + zo, *vt = sm + L::UT + i + zo;
#pragma unroll 2
            for (int j = 0; j < 8; j++) {
                const float v = zc[j * 6];
                at += div64((2.f * v) * vt[j * zs], C.id2z64);
                an += div64(v * vn[j * zs], C.id2z64);
            }
        } else {
            const Brk b = brackets(sm + L::MU + i, 1);
            if (VTI && !XB) at = d2i(at, brackets(sm + L::Q + i, 1), sm + L::UT + i, 1, inv_d2t);
            else at = d2i(at, twice(b), sm + L::UT + i, 1, inv_d2t);
            an = d2i(an, b, sm + L::UN + i, 1, inv_d2t);
        }
#pragma unroll
        for (int j = 0; j < 8; j++) at += div64(CL[j * kFusedBand] * UT[j * kFs], idn2);
        // mixed terms
        if (VTI) {
            an += dern(L::D);
            at += dert(L::D1);
        } else {
            an += mdern(L::D, L::Q);
            at += mdert(AE ? L::D1 : L::D, L::Q);
        }
        if (AE) {
            an += mdern(L::D1, L::Q);
            at += mdert(L::D, L::Q);
        }
        if (XB) {
            at += mdern(L::DT, L::MU);
            an += mdert(L::DS, L::MU);
        } else {
            an += mdert(L::DS, L::MU);
            at += mdern(L::DT, L::MU);
        }
        // sources of this cell, in the reference's order
        // (its entries: first, then the counts of ux and uz entries)
        const int nx_ = __float_as_int(SF[SL_NX * kFt]), nz_ = __float_as_int(SF[SL_NZ * kFt]);
        if (nx_ + nz_ > 0) {
            const int e = __float_as_int(SF[SL_E0 * kFt]);
            auto value = [&](int k) {
                if (cached) return sm[L::VAL + k];
                const InjEntry &E = Sp->inj[inj0 + k];
                return E.mt ? (E.wa * srcrow[E.ia] - E.wb * srcrow[E.ib]) : E.wa * srcrow[E.ia];
            };
            for (int k = 0; k < nx_; k++) {
                if (XB) an += value(e + k);
                else at += value(e + k);
            }
            for (int k = 0; k < nz_; k++) {
                if (XB) at += value(e + nx_ + k);
                else an += value(e + nx_ + k);
            }
        }
    }
    __syncthreads();   // the SAT terms of warps 6 and 7

    if (owned) {
        // subtracted in the reference's side order: top, bottom, left, right (the fluid
        // interface of the acoustic-elastic propagator, its top edge, last)
        auto corner = [&](int side) {
            const int bc = side == 0 ? C.bc[0] : C.bc[1];
            if (bc != 1 && bc != 2) return;
            const float *q = sm + L::SAT + 96 + warp;
            an = an - q[0];
            at = at - q[32];
            at = at - q[64];
        };
        if (XB && !AE && gz == 0) corner(0);
        if (XB && gz == nz - 1) corner(1);
        if (warp == 0) {
            const int bc = br.side == 0 ? C.bc[0] : br.side == 1 ? C.bc[1] : br.side == 2 ? C.bc[2] : C.bc[3];
            if (bc == 1 || bc == 2) {
                const float *q = sm + L::SAT + lane;
                at = at - q[0];
                an = an - q[32];
                an = an - q[64];
            }
        }
        if (XB && AE && gz == 0) corner(0);

        const double irho = SD[0];
        an = div64(C.dt2 * an, irho) + 2 * un - pn_;
        at = div64(C.dt2 * at, irho) + 2 * ut - pt_;
        float n0 = XB ? an : at, n1 = XB ? at : an;
        if (edge) {
            n0 = div64(n0, SD[kFt]);
            n1 = div64(n1, SD[2 * kFt]);
        }
        n0 = n0 * tzv * txv;
        if (AE && gz == 0) Sp->halo_save[gx] = XB ? pt_ : pn_;   // interface row: coupled and tapered by ae_couple
        else n1 = n1 * tzv * txv;
        pn[cell] = n0;
        pn[nxz + cell] = n1;
        amax = fmaxf(fabsf(n0), fabsf(n1));
        const int slot = by(it, C.sub);
        if (!GRAD && (A.flags & F_STORE) && slot * C.sub == it) {
            const float sc = prec == SNAP_FP32 ? 1.f : snap_scale(Sp->snap_amax, slot);
            const long long o = (long long)slot * Sp->snap_slot + cell;
            snap_store(Sp->snap, o, prec, XB ? un : ut, sc);
            snap_store(Sp->snap, o + nxz, prec, XB ? ut : un, sc);
        }

        if (GRAD && do_grad) {
            // strains of the adjoint field (this thread's own) and of the snapshot
            const float ax0 = XB ? en : et, az1 = XB ? et : en, ax1 = XB ? es : eq, az0 = XB ? eq : es;
            const int F0 = L::snap(itf, 0), F1 = L::snap(itf, 1), FN = XB ? F0 : F1, FT = XB ? F1 : F0;
            const float qn = dern(FN), qt = dert(FT), qs = dern(FT), qq = dert(FN);
            const float q0 = XB ? qn : qt, q1 = XB ? qt : qn, q2 = XB ? qs : qq, q3 = XB ? qq : qs;
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
                G[2 * (long long)nxz] = density_term(g2, wdt, itf, last, n0, n1, sm[F0 + i], sm[F1 + i],
                                                     sm[L::snap(itf + 1, 0) + i], sm[L::snap(itf + 1, 1) + i],
                                                     sm[L::snap(itf - 1, 0) + i], sm[L::snap(itf - 1, 1) + i]);
        }
    }
    if (!GRAD && (A.flags & F_AMAX) && (it + 1) % C.sub == 0)
        block_amax(amax, sm + L::RED, Sp->snap_amax + (it + 1) / C.sub);
    return true;
}

// ---------------------------------------------------------------------------
// Acoustic unit: a window of 32 (z) x 16 (x) cells of a shot's pressure (or of
// the fluid layer's potential, FLUID), the tile kernel's windows and arithmetic
// (acoustic.cuh, src/cpp/we_op.cpp:1937-2134).  Windows clear of the closures
// take the z-pair form of the elastic windows; the others are cut into units of
// 8 columns (their owned cells), one cell per thread through the general forms:
// such a unit's time is one thread's chain, which sets the step on small plans.
// ---------------------------------------------------------------------------
template <bool GRAD>
struct AcLayout {
    static constexpr int U = 0, IR = kFu, F = IR + kFw, VAL = F + (GRAD ? kFw : 0), KEY = VAL + kVal;
    static constexpr int RED = KEY + kVal, FLOATS = RED + 8;
};

// imaging condition of one cell at the start of a step (nl_we_op_a::compute_gradients, we_op.cpp:1883-1935)
__device__ __forceinline__ void acoustic_image(float &g0, float &g1, float t0, float t1, float t2, float t3, float f, float adj,
                                               float K, float fp, float fm, float w, float dtg, int itf, int last)
{
    const double c = (double)w * 1.0 / (double)(dtg * K * K) * (double)adj;
    const float s = itf > 0 && itf < last ? fp - 2 * f + fm : itf == 0 ? fp - f : -f + fm;
    g0 = (float)((double)g0 - c * (double)s);
    if (itf == 0) g1 = (float)((double)g1 + (double)w * 0.5 * (double)dtg * (double)(t2 * t0 + t3 * t1));
    else g1 += w * dtg * (t2 * t0 + t3 * t1);
}

template <bool GRAD, bool FLUID, class Meet>
__device__ __forceinline__ bool acoustic_unit(const ShotDev *__restrict__ Sp, const ModelDev &M, const StepConst &C,
                                              const TileRef tr, const int it, const int flags, const float dtg,
                                              const bool keep, float *sm, Meet meet_first)
{
    using L = AcLayout<GRAD>;
    const int t = threadIdx.x, nt = Sp->nt, nx = Sp->nx, nz = Sp->nz, ldz = Sp->ldz, mld = M.ldz;
    const int wx0 = tr.wx0, wz0 = tr.wz0, prec = C.snap_prec;
    const long long mofs = (long long)Sp->x0 * mld, nxz = (long long)nx * ldz;
    const bool inner = wx0 >= 6 && wx0 + kFx + 6 <= nx && wz0 >= 6 && wz0 + kFz + 6 <= nz && (wz0 & 3) == 0;
    // snapshot (nt-1-it)/sub, skipped at it == 0 (we_op.cpp:2044-2046)
    const int kk = nt - 1 - it, itf = GRAD ? by(kk, C.sub) : 0, last = by(nt, C.sub);
    const bool do_grad = GRAD && it != 0 && kk > 0 && itf * C.sub == kk;
    float finv = 1.f;
    if (GRAD && do_grad && prec != SNAP_FP32) finv = 1.f / snap_scale(Sp->snap_amax, itf);
    const int xr = t / 10, xq = 4 * (t - 10 * xr);

    // ---- what no step writes
    if (inner) {
        if (t < (kFx + 4) * 10) {
            const int s = xr * kFs + xq;
            if (!keep) cp16(sm + L::IR + s, M.p1 + mofs + (long long)(wx0 - 2 + xr) * mld + wz0 - 4 + xq, true);
            if (GRAD && do_grad) {
                const long long so = (long long)itf * Sp->snap_slot + (long long)(wx0 - 2 + xr) * ldz + wz0 - 4 + xq;
                if (prec == SNAP_FP32) cp16(sm + L::F + s, (const float *)Sp->snap + so, true);
                else *reinterpret_cast<float4 *>(sm + L::F + s) = snap_load4(Sp->snap, so, prec, finv);
            }
        }
    } else {
        for (int i = t; i < kFw; i += kFt) {
            const int r = i / kFs, q = i - r * kFs, x = wx0 - 2 + r, z = wz0 - 4 + q;
            const bool in = x >= 0 && x < nx && z >= 0 && z < nz;
            if (!keep) sm[L::IR + i] = in ? M.p1[mofs + (long long)x * mld + z] : 0.f;
            if (GRAD && do_grad)
                sm[L::F + i] = in ? snap_load(Sp->snap, (long long)itf * Sp->snap_slot + (long long)x * ldz + z, prec, finv) : 0.f;
        }
    }
    // this step's injected values and their cells (sorted by cell, the reference's order within one)
    const int inj0 = Sp->inj_off[tr.unit], ninj = Sp->inj_off[tr.unit + 1] - inj0;
    const float *srcrow = Sp->src + (long long)it * Sp->nsrc;
    if (it < nt - 1 && ninj <= kVal)
        for (int e = t; e < ninj; e += kFt) {
            const InjEntry &E = Sp->inj[inj0 + e];
            sm[L::VAL + e] = E.wa * srcrow[E.ia];
            sm[L::KEY + e] = __int_as_float((E.gx - wx0) * kFz + E.gz - wz0);
            asm volatile("prefetch.global.L2 [%0];" ::"l"(srcrow + Sp->nsrc + E.ia));
        }
    auto value = [&](int e) {
        if (ninj <= kVal) return sm[L::VAL + e];
        const InjEntry &E = Sp->inj[inj0 + e];
        return E.wa * srcrow[E.ia];
    };
    auto key = [&](int e) {
        if (ninj <= kVal) return __float_as_int(sm[L::KEY + e]);
        const InjEntry &E = Sp->inj[inj0 + e];
        return (E.gx - wx0) * kFz + E.gz - wz0;
    };
    auto first_entry = [&](int k) {   // of the cells from k on
        int lo = 0, hi = ninj;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (key(mid) < k) lo = mid + 1;
            else hi = mid;
        }
        return lo;
    };
    // general form: this thread's cell and what it needs of the model
    const int half = (tr.ox0 - wx0) >> 3, ctz = t & 31, ctx = (t >> 5) + 8 * half, cgx = wx0 + ctx, cgz = wz0 + ctz;
    const bool cown = !inner && cgx >= tr.ox0 && cgx < tr.ox1 && cgz >= tr.oz0 && cgz < tr.oz1;
    // closure coefficients of the axis (0 x, 1 z) at this cell
    auto closure = [&](int ax, float (&v)[8]) {
        const int g = ax ? cgz : cgx, na = ax ? nz : nx, ld = ax ? M.nx : ldz;
        const bool far = g >= 6;
        const float *cl = (ax ? M.zclos + Sp->x0 + cgx : Sp->xclos + cgz) +
                          (long long)((far ? 48 : 0) + (far ? na - 1 - g : g) * 8) * ld;
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = cl[(long long)j * ld];
    };
    const bool cx = cown && (cgx < 6 || cgx >= nx - 6), cz = cown && (cgz < 6 || cgz >= nz - 6);
    float K = 0.f, tzv = 0.f, txv = 0.f, v[8];
    if (cown) {
        K = M.p0[mofs + (long long)cgx * mld + cgz];
        tzv = Sp->tz[cgz];
        txv = Sp->tx[cgx];
        if (cx || cz) closure(cx ? 0 : 1, v);
    }
    const float *curr = Sp->u[(it + 1) & 1];
    float *pn = Sp->u[it & 1];
    if (!meet_first()) {
        cp_wait();
        return false;
    }
    if (it >= nt - 1) {
        cp_wait();
        return true;
    }
    if (inner) {
        if (t < (kFx + 8) * 10)
            cp16(sm + L::U + xr * kFs + xq, curr + (long long)(wx0 - 4 + xr) * ldz + wz0 - 4 + xq, true);
        cp_wait();
    } else {
        float w[4];
#pragma unroll
        for (int h = 0; h < 4; h++) {
            const int i = t + h * kFt, r = i / kFs, q = i - r * kFs, x = wx0 - 4 + r, z = wz0 - 4 + q;
            w[h] = i < kFu && x >= 0 && x < nx && z >= 0 && z < nz ? __ldcg(curr + (long long)x * ldz + z) : 0.f;
        }
#pragma unroll
        for (int h = 0; h < 4; h++)
            if (t + h * kFt < kFu) sm[L::U + t + h * kFt] = w[h];
    }
    __syncthreads();

    const float *U = sm + L::U + 2 * kFs, *IR = sm + L::IR, *F = sm + L::F;   // one index for all
    // receivers of the tile: a cut tile's first half takes them all (every tile has one, its window covers both)
    if (!GRAD && (flags & F_EXTRACT) && (inner || half == 0)) {
        const int r1 = Sp->ext_off[tr.unit + 1];
        for (int e = Sp->ext_off[tr.unit] + t; e < r1; e += kFt) {
            const ExtEntry &E = Sp->ext[e];
            const float *u = sm + L::U + (E.gx0 - wx0 + 4) * kFs + (E.gz0 - wz0 + 4);
            float o = 0.f;
#pragma unroll
            for (int a = 0; a < 3; a++)
#pragma unroll
                for (int b = 0; b < 3; b++) o += E.w[a * 3 + b] * u[a * kFs + b];
            Sp->rcv[(long long)it * Sp->nrcv + E.row] = o;
        }
    }
    const int slot = by(it, C.sub);
    const bool store = !GRAD && (flags & F_STORE) && slot * C.sub == it;
    float amax = 0.f;

    if (inner) {
        const int tx = t >> 4, pz = 2 * (t & 15), gx = wx0 + tx, gz = wz0 + pz, i = (tx + 2) * kFs + 4 + pz;
        const bool ownx = gx >= tr.ox0 && gx < tr.ox1;
        const bool own0 = ownx && gz >= tr.oz0 && gz < tr.oz1, own1 = ownx && gz + 1 >= tr.oz0 && gz + 1 < tr.oz1;
        const long long cell = (long long)gx * ldz + gz;
        const float2 p = __ldcg(reinterpret_cast<const float2 *>(pn + cell));
        const float2 K2 = *reinterpret_cast<const float2 *>(M.p0 + mofs + (long long)gx * mld + gz);
        const float2 tz2 = *reinterpret_cast<const float2 *>(Sp->tz + gz), tzx = bc2(Sp->tx[gx]);
        const float2 um2 = ld2(U, i - 2 * kFs), um1 = ld2(U, i - kFs), u0 = ld2(U, i), up1 = ld2(U, i + kFs),
                     up2 = ld2(U, i + 2 * kFs), ulo = ld2(U, i - 2), uhi = ld2(U, i + 2);
        if (GRAD && do_grad && (own0 || own1)) {
            const float2 f = ld2(F, i);
            const float2 t0 = der_x(ld2(F, i - 2 * kFs), ld2(F, i - kFs), ld2(F, i + kFs), ld2(F, i + 2 * kFs), C.sdx);
            const float2 t1 = der_z(ld2(F, i - 2), f, ld2(F, i + 2), C.sdz);
            const float2 t2 = der_x(um2, um1, up1, up2, C.sdx), t3 = der_z(ulo, u0, uhi, C.sdz);
            float2 fp = make_float2(0.f, 0.f), fm = fp;
            if (itf + 1 <= last) {
                const float inv = prec == SNAP_FP32 ? 1.f : 1.f / snap_scale(Sp->snap_amax, itf + 1);
                fp = snap_load2(Sp->snap, (long long)(itf + 1) * Sp->snap_slot + cell, prec, inv);
            }
            {
                const float inv = prec == SNAP_FP32 ? 1.f : 1.f / snap_scale(Sp->snap_amax, itf - 1);
                fm = snap_load2(Sp->snap, (long long)(itf - 1) * Sp->snap_slot + cell, prec, inv);
            }
            const float w = Sp->gwt[itf];
            float *g = Sp->grad + cell;
            float2 g0 = __ldcg(reinterpret_cast<const float2 *>(g)), g1 = __ldcg(reinterpret_cast<const float2 *>(g + nxz));
            acoustic_image(g0.x, g1.x, t0.x, t1.x, t2.x, t3.x, f.x, u0.x, K2.x, fp.x, fm.x, w, dtg, itf, last);
            acoustic_image(g0.y, g1.y, t0.y, t1.y, t2.y, t3.y, f.y, u0.y, K2.y, fp.y, fm.y, w, dtg, itf, last);
            if (own0) {
                g[0] = g0.x;
                g[nxz] = g1.x;
            }
            if (own1) {
                g[1] = g0.y;
                g[nxz + 1] = g1.y;
            }
        }
        const float2 r00 = ld2(IR, i), rlo = ld2(IR, i - 2), rhi = ld2(IR, i + 2);
        const Brk2 bx = brackets2(ld2(IR, i - 2 * kFs), ld2(IR, i - kFs), r00, ld2(IR, i + kFs), ld2(IR, i + 2 * kFs));
        float2 n = mul2(bc2(C.inv_d2x), sum_x(bx, um2, um1, u0, up1, up2));
        const Brk2 bz = brackets2(rlo, zsh(rlo, r00), r00, zsh(r00, rhi), rhi);
        n = add2(n, mul2(bc2(C.inv_d2z), sum_z(bz, ulo, u0, uhi)));
        if (ninj > 0) {
            const int k = tx * kFz + pz;
            for (int e = first_entry(k); e < ninj && key(e) <= k + 1; e++) {
                if (key(e) == k) n.x += value(e);
                else n.y += value(e);
            }
        }
        float2 q = p;
        if (it > 0) q = mul2(mul2(q, tz2), tzx);
        // dt^2 n K + 2 curr - prev, tapered
        n = dif2(fma2(bc2(2.f), u0, mul2(mul2(bc2(C.dt2), n), K2)), q);
        n = mul2(mul2(n, tz2), tzx);
        if (own0) pn[cell] = n.x;
        if (own1) pn[cell + 1] = n.y;
        if (store) {
            const float sc = prec == SNAP_FP32 ? 1.f : snap_scale(Sp->snap_amax, slot);
            const long long o = (long long)slot * Sp->snap_slot + cell;
            if (own0) snap_store(Sp->snap, o, prec, u0.x, sc);
            if (own1) snap_store(Sp->snap, o + 1, prec, u0.y, sc);
        }
        if (own0) amax = fabsf(n.x);
        if (own1) amax = fmaxf(amax, fabsf(n.y));
    } else if (cown) {
        {
            const int gx = cgx, gz = cgz, i = (ctx + 2) * kFs + 4 + ctz;
            const long long cell = (long long)gx * ldz + gz;
            const float u0 = U[i];
            float p = __ldcg(pn + cell);
            if (store) {
                const float sc = prec == SNAP_FP32 ? 1.f : snap_scale(Sp->snap_amax, slot);
                snap_store(Sp->snap, (long long)slot * Sp->snap_slot + cell, prec, u0, sc);
            }
            if (GRAD && do_grad) {
                const float t0 = d1(F + i, kFs, gx, nx, C.dx, C.sdx), t1 = d1(F + i, 1, gz, nz, C.dz, C.sdz);
                const float t2 = d1(U + i, kFs, gx, nx, C.dx, C.sdx), t3 = d1(U + i, 1, gz, nz, C.dz, C.sdz);
                float fp = 0.f, fm = 0.f;
                if (itf + 1 <= last) {
                    const float inv = prec == SNAP_FP32 ? 1.f : 1.f / snap_scale(Sp->snap_amax, itf + 1);
                    fp = snap_load(Sp->snap, (long long)(itf + 1) * Sp->snap_slot + cell, prec, inv);
                }
                {
                    const float inv = prec == SNAP_FP32 ? 1.f : 1.f / snap_scale(Sp->snap_amax, itf - 1);
                    fm = snap_load(Sp->snap, (long long)(itf - 1) * Sp->snap_slot + cell, prec, inv);
                }
                float *g = Sp->grad + cell;
                float g0 = __ldcg(g), g1 = __ldcg(g + nxz);
                acoustic_image(g0, g1, t0, t1, t2, t3, F[i], u0, K, fp, fm, Sp->gwt[itf], dtg, itf, last);
                g[0] = g0;
                g[nxz] = g1;
            }
            float n = 0.f;
            // second derivative along x, then z
#pragma unroll
            for (int ax = 0; ax < 2; ax++) {
                const int g = ax ? gz : gx, na = ax ? nz : nx, st = ax ? 1 : kFs;
                if (!(ax ? cz : cx)) {
                    n = d2i(n, brackets(IR + i, st), U + i, st, ax ? C.inv_d2z : C.inv_d2x);
                    continue;
                }
                if (ax && cx) closure(1, v);   // a corner cell
                const bool far = g >= 6;
                const int in = far ? -st : st;
                const float *u = U + i + (far ? na - 1 - g : -g) * st;
#pragma unroll
                for (int j = 0; j < 8; j++) n += div64(v[j] * u[j * in], ax ? C.id2z64 : C.id2x64);
            }
            if (ninj > 0) {
                const int k = ctx * kFz + ctz;
                for (int e = first_entry(k); e < ninj && key(e) == k; e++) n += value(e);
            }
            if (it > 0) p = p * tzv * txv;
            // sides in the reference's order: top, bottom, left, right (the fluid's interface, its bottom, last)
#pragma unroll 1
            for (int k = 0; k < 4; k++) {
                const int side = !FLUID ? k : (k == 0 ? 0 : k == 3 ? 1 : k + 1);
                const int bc = side == 0 ? C.bc[0] : side == 1 ? C.bc[1] : side == 2 ? C.bc[2] : C.bc[3];
                const int dist = side == 0 ? gz : side == 1 ? nz - 1 - gz : side == 2 ? gx : nx - 1 - gx;
                if (bc < 1 || bc > 3 || dist >= 4) continue;
                const int st = side == 0 ? 1 : side == 1 ? -1 : side == 2 ? kFs : -kFs;
                n = asat_cell(n, side, bc, dist, U + i, st, IR + i, st, p, K, C);
            }
            n = C.dt2 * n * K + 2 * u0 - p;
            if (gz == 0 || gz == nz - 1 || gx == 0 || gx == nx - 1) {
                const int q = gz == 0 ? gx : gz == nz - 1 ? nx + gx : gx == 0 ? 2 * nx + gz : 2 * nx + nz + gz;
                if (n != 0.f) n = n / Sp->den[q];   // den > 0
            }
            if (FLUID && gz == nz - 1) Sp->halo_save[gx] = p;   // interface row: coupled and tapered there
            else n = n * tzv * txv;
            pn[cell] = n;
            amax = fmaxf(amax, fabsf(n));
        }
    }
    if (!GRAD && !FLUID && (flags & F_AMAX) && (it + 1) % C.sub == 0)
        block_amax(amax, sm + L::RED, Sp->snap_amax + (it + 1) / C.sub);
    return true;
}

struct AcousticArgs {
    const ShotDev *shots;
    const TileRef *tiles;
    int ntile;
    ModelDev M;
    StepConst C;
    int it0, it1, flags;
    float dtg;
    unsigned *count;
    int *status;
};

// The time loop of the acoustic propagator.  Bound by the tiles beside a closure
// (general forms, double-precision quotients), which 8-column units keep short:
// three 401 x 301 shots 23 / 30 us a step forward / adjoint in launches per step,
// 11.5 / 19.1 here.  Four CTAs per SM: the adjoint takes 21.4 us with three (its
// units are many more than the CTAs), the forward 17.2 with five;
// one 201 x 151 shot, a tile per CTA, 7.88 us and 7.76 with three.
template <bool GRAD>
__global__ void __launch_bounds__(kFt, 4) acoustic_steps(const __grid_constant__ AcousticArgs A)
{
    extern __shared__ __align__(1024) float sm[];
    const int G = gridDim.x;
    for (int it = A.it0; it < A.it1; it++) {
        for (int u = blockIdx.x; u < A.ntile; u += G) {
            const TileRef tr = A.tiles[u];
            const bool first = u == (int)blockIdx.x, keep = (int)blockIdx.x + G >= A.ntile && it > A.it0;
            if (!acoustic_unit<GRAD, false>(A.shots + tr.shot, A.M, A.C, tr, it, A.flags, A.dtg, keep, sm, [&]() {
                    return !first || meet_at(A.count, A.status, A.C.spin, (unsigned)(it - A.it0), it);
                }))
                return;
            __syncthreads();
        }
        if (threadIdx.x == 0 && it + 1 < A.it1) arrive(A.count);
    }
}

// Table entries of the windows to come, copied ahead: the next window's shot and
// the tile after it (whose address needs nothing that is still on its way).
__device__ __forceinline__ void fetch16(void *dst, const void *src, int bytes, int lane0)
{
    const int q = (int)threadIdx.x - lane0;
    if (q >= 0 && q < bytes / 16) cp16((float *)dst + 4 * q, (const float *)src + 4 * q, true);
}

// BLOCKS: resident CTAs per SM asked of the compiler.  The adjoint's shared memory
// allows four (VTI: three).  The forward takes five (48 registers, a few spills)
// where there are units for them, and four (64 registers) where each CTA has its
// one unit anyway and a step lasts as long as a band unit's chain of
// instructions: 8 shots of 801 x 401 52.1 -> 45.7 us a step with five, but one
// 81 x 61 shot 5.9 -> 6.4 us.
template <bool VTI, bool GRAD, bool AE, bool S16, int BLOCKS>
__global__ void __launch_bounds__(kFt, BLOCKS)
fused_steps(const __grid_constant__ FusedArgs A)
{
    extern __shared__ __align__(1024) float sm[];
    static_assert(sizeof(ShotDev) % 16 == 0 && sizeof(WinRef) % 16 == 0, "copied in 16-byte pieces");
    __shared__ __align__(16) ShotDev S_[2];
    __shared__ __align__(16) WinRef T_[4];
    const int G = gridDim.x;
    // slots blockIdx.x, + G, ... of the units (band units first) rotated so that, with
    // fewer than two units per CTA, the band units (the longest) get a CTA of their own
    const int off = A.nunit < 2 * G ? max(0, A.nunit - G) : 0;
    auto unit = [&](int m) {
        const int slot = blockIdx.x + m * G;
        return slot >= off ? slot - off : slot - off + A.nunit;
    };
    const int n = (A.nunit - (int)blockIdx.x + G - 1) / G;   // this CTA's units
    // its only unit (a tile of the fluid layer would take the same shared memory)
    const bool one = n == 1 && !(AE && G - 1 - (int)blockIdx.x < A.W.ntile);
    // its windows are the slots [w0, w0 + nw), the others are band units
    int w0 = 0, nw = 0;
    for (int m = 0; m < n; m++)
        if (unit(m) >= A.nband) {
            if (nw == 0) w0 = m;
            nw++;
        }
    auto window = [&](int q) { return A.in + (unit(w0 + q % nw) - A.nband); };
    int q = 0;   // windows done so far
    unsigned par_lead = 0, par_own = 0;
    bool ring = false;
    __shared__ unsigned long long bars[2];
    __shared__ float inv_[2][3];   // S16: factors of the snapshots before, at and after the imaging time
    unsigned long long *const lead = bars, *const own = bars + 1;
    if (nw > 0) {
        if (threadIdx.x == 0) {
            bar_init(lead);
            bar_init(own);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        fetch16(&T_[0], window(0), sizeof(WinRef), 0);
        fetch16(&T_[1], window(1), sizeof(WinRef), 32);
        fetch16(&S_[0], A.shots + window(0)->shot, sizeof(ShotDev), 64);
        cp_wait();
        __syncthreads();
    }
    for (int it = A.it0; it < A.it1; it++) {
        const bool keep = one && it > A.it0;
        bool first = true;
        for (int m = 0; m < n; m++) {
            if (nw > 0 && m >= w0 && m < w0 + nw) continue;
            const BandRef br = A.bands[unit(m)];
            const bool ok = br.side >= 2 ? fused_band<true, VTI, GRAD, AE>(A, br, it, first, keep, one, ring, sm)
                                         : fused_band<false, VTI, GRAD, AE>(A, br, it, first, keep, one, ring, sm);
            if (!ok) return;
            first = false;
            __syncthreads();
        }
        if (AE) {
            // tiles of the fluid layer, from the last CTA on
            for (int u = G - 1 - (int)blockIdx.x; u < A.W.ntile; u += G) {
                const TileRef tr = A.W.tiles[u];
                if (!acoustic_unit<false, true>(A.W.shots + tr.shot, A.W.M, A.W.C, tr, it, A.flags & F_EXTRACT, 1.f, false, sm,
                                                [&]() { return !first || meet<AE>(A, it); }))
                    return;
                first = false;
                __syncthreads();
            }
        }
        for (int k = 0; k < nw; k++, q++) {
            const ShotDev &S = S_[q & 1], &Sn = S_[(q + 1) & 1];
            const WinRef &tr = T_[q & 3], &tn = T_[(q + 1) & 3];
            const bool active = it < S.nt - 1;
            if (k == 0) {
                // the first window of a step: what no step writes, then the meeting, then the fields
                if (active) {
                    if (threadIdx.x == 0) {
                        fence_async();
                        bar_expect(lead, lead_bytes<VTI>(!keep));
                        issue_lead<VTI, GRAD, AE>(A, S, tr, it, !keep, false, sm, lead);
                        issue_own_static<VTI, GRAD, AE>(A, S, tr, it, !keep, sm, own);
                    }
                    if (S16) set_factors(S, imaging<GRAD, AE>(S, A.C, it), inv_[q & 1]);
                }
                if (first && !meet<AE>(A, it, [&]() { finish_copies<GRAD, AE>(A, S, it, bars); })) return;
                if (active && threadIdx.x == 0) {
                    fence_async();
                    issue_lead<VTI, GRAD, AE>(A, S, tr, it, false, true, sm, lead);
                    issue_own_fields<VTI, GRAD, AE>(A, S, tr, it, sm, own);
                }
            }
            fetch16(&T_[(q + 2) & 3], window(q + 2), sizeof(WinRef), 32);
            fetch16(&S_[(q + 1) & 1], A.shots + tn.shot, sizeof(ShotDev), 64);
            // between the halves: the Own group and the next entries have arrived, all
            // threads have left the first half
            auto ahead = [&](bool lead_ok) {
                const bool ok = !active || (wait_bar(A, own, par_own, it) && lead_ok);
                cp_wait();
                if (__syncthreads_or(!ok)) return false;
                if (k + 1 < nw && it < Sn.nt - 1 && threadIdx.x == 0) {
                    fence_async();
                    bar_expect(lead, lead_bytes<VTI>(true));
                    issue_lead<VTI, GRAD, AE>(A, Sn, tn, it, true, true, sm, lead);
                }
                return true;
            };
            if (active) {
                if (!window_step<VTI, GRAD, AE, S16>(
                        A, S, tr, it, sm, inv_[q & 1], [&]() { return wait_bar(A, lead, par_lead, it); }, ahead))
                    return;
            } else if (!ahead(true)) {
                return;
            }
            if (k + 1 == nw) fence_async();   // this step's writes, before the arrival
            __syncthreads();
            if (k + 1 < nw && it < Sn.nt - 1) {
                if (threadIdx.x == 0) {
                    fence_async();
                    issue_own_static<VTI, GRAD, AE>(A, Sn, tn, it, true, sm, own);
                    issue_own_fields<VTI, GRAD, AE>(A, Sn, tn, it, sm, own);
                }
                if (S16) set_factors(Sn, imaging<GRAD, AE>(Sn, A.C, it), inv_[(q + 1) & 1]);
            }
        }
        if (nw == 0) {
            if (AE && first && !meet<AE>(A, it)) return;
            fence_async();
            __syncthreads();
        }
        if (AE) {
            // the coupling of fluid and elastic rows, column by column
            if (threadIdx.x == 0) arrive(A.count);
            if (!meet_at(A.count, A.status, A.C.spin, 2u * (unsigned)(it - A.it0) + 1u, it)) return;
            const int per = (A.W.ncol + kFt - 1) / kFt;
            for (int c = blockIdx.x; c < per * A.W.nshot; c += G) {
                const int sh = A.W.s0 + c / per;
                ae_couple_column(A.shots[sh], A.W.shots[sh], (c % per) * kFt + threadIdx.x, A.M, A.C, it, A.flags, A.dtg,
                                 A.W.Kw, A.W.val0, A.W.sign);
            }
            fence_async();
            __syncthreads();
        }
        if (threadIdx.x == 0 && it + 1 < A.it1) arrive(A.count);
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

void upload_fused_tables(const float *b1, const float *b2, const float *c2, const float *c1, const float *sc,
                         const float *hc)
{
    cudaMemcpyToSymbol(kHC, hc, sizeof(float) * 4);
    cudaMemcpyToSymbol(kB1, b1, sizeof(float) * 24);
    cudaMemcpyToSymbol(kB2, b2, sizeof(float) * 384);
    cudaMemcpyToSymbol(kC2, c2, sizeof(float) * 10);
    cudaMemcpyToSymbol(kC1, c1, sizeof(float) * 2);
    cudaMemcpyToSymbol(kSC, sc, sizeof(float) * 4);
    const float2 one = make_float2(1.f, 1.f), minus = make_float2(-1.f, -1.f);
    cudaMemcpyToSymbol(kOne2, &one, sizeof(one));
    cudaMemcpyToSymbol(kMinus2, &minus, sizeof(minus));
}

// A cooperative launch of at most the resident CTAs over `units`.
template <class Args>
static cudaError_t launch_loop(void (*kernel)(const Args), const Args &A, int units, size_t bytes, unsigned *count,
                               cudaStream_t st)
{
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    int dev = 0, sms = 0, per = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, kFt, bytes);
    if (e == cudaSuccess) e = cudaMemsetAsync(count, 0, sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    const long long room = (long long)sms * per;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(units < room ? units : room));
    cfg.blockDim = dim3(kFt);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;   // all CTAs resident: they wait for one another
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, A);
}

template <bool VTI, bool GRAD, bool AE>
static cudaError_t launch_fused_t(const FusedArgs &A, cudaStream_t st)
{
    constexpr size_t bytes = fused_bytes<VTI, GRAD, AE>();
    if constexpr (GRAD) {
        constexpr int blocks = VTI ? 3 : 4;
        if (A.C.snap_prec != SNAP_FP32)
            return launch_loop(fused_steps<VTI, GRAD, AE, true, blocks>, A, A.nunit, bytes, A.count, st);
        return launch_loop(fused_steps<VTI, GRAD, AE, false, blocks>, A, A.nunit, bytes, A.count, st);
    } else {
        int dev = 0, sms = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        if (A.nunit <= 4 * sms) return launch_loop(fused_steps<VTI, GRAD, AE, false, 4>, A, A.nunit, bytes, A.count, st);
        return launch_loop(fused_steps<VTI, GRAD, AE, false, 5>, A, A.nunit, bytes, A.count, st);
    }
}

// ---- tensor maps ----------------------------------------------------------------
// cuTensorMapEncodeTiled through the runtime (the library does not link the driver)
static cudaError_t encode(CUtensorMap *m, const void *base, int rank, const cuuint64_t *dim, const cuuint32_t *box,
                          bool half = false)
{
    if ((size_t)m % alignof(CUtensorMap)) return cudaErrorMisalignedAddress;   // the driver's rule, for the host copy too
    using Fn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                            const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                            CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    const cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q);
    if (e != cudaSuccess) return e;
    if (!f || q != cudaDriverEntryPointSuccess) return cudaErrorNotSupported;
    cuuint64_t stride[3];
    cuuint32_t one[4] = {1, 1, 1, 1};
    cuuint64_t s = half ? 2 : 4;
    for (int i = 0; i + 1 < rank; i++) stride[i] = s *= dim[i];
    const CUresult r = ((Fn)f)(m, half ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, rank, const_cast<void *>(base), dim, stride, box, one,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

size_t fused_maps_bytes() { return SM_COUNT * sizeof(CUtensorMap); }

cudaError_t fused_shot_maps(void *out, int nx, int ldz, const float *u0, const float *u1, const float *grad,
                            const void *snap, int nslot, bool half)
{
    CUtensorMap m[SM_COUNT];   // aligned as the driver asks, which `out` need not be
    static_assert(alignof(CUtensorMap) == 64, "alignment of a tensor map");
    std::memset(m, 0, sizeof(m));
    const cuuint64_t d2[3] = {(cuuint64_t)ldz, (cuuint64_t)nx, 2}, d3[3] = {(cuuint64_t)ldz, (cuuint64_t)nx, 3};
    const cuuint64_t ds[4] = {(cuuint64_t)ldz, (cuuint64_t)nx, 2, (cuuint64_t)nslot};
    const cuuint32_t lead[3] = {kFs, kFx + 8, 2}, own[4] = {kFz, kFx, 2, 1}, g[3] = {kFz, kFx, 3}, sl[4] = {kFs, kFx + 4, 2, 1};
    cudaError_t e = cudaSuccess;
    const float *u[2] = {u0, u1};
    for (int b = 0; b < 2 && e == cudaSuccess; b++) {
        e = encode(m + SM_LEAD + b, u[b], 3, d2, lead);
        if (e == cudaSuccess) e = encode(m + SM_OWN + b, u[b], 3, d2, own);
    }
    if (e == cudaSuccess && grad) e = encode(m + SM_GRAD, grad, 3, d3, g);
    if (e == cudaSuccess && snap && nslot > 0) {
        // 16-bit: the own cells from the window's first sample but four on, a multiple of 16 bytes
        const cuuint32_t raw[4] = {kFs, kFx, 2, 1};
        e = encode(m + SM_SNAP_LEAD, snap, 4, ds, sl, half);
        if (e == cudaSuccess) e = encode(m + SM_SNAP_OWN, snap, 4, ds, half ? raw : own, half);
    }
    std::memcpy(out, m, sizeof(m));
    return e;
}

static cudaError_t model_maps(CUtensorMap *m, int kind, const ModelDev &M)
{
    const cuuint64_t dim[2] = {(cuuint64_t)M.ldz, (cuuint64_t)M.nx};
    const cuuint32_t halo[2] = {kFs, kFx + 4}, own[2] = {kFz, kFx};
    const bool vti = kind == KIND_VTI;
    const float *p[MM_COUNT] = {M.p1, vti ? M.fxx : M.p0, M.lbis, M.c13, M.p0, M.p2, M.irho, M.eps, M.gv2, M.gv3};
    for (int i = 0; i < MM_COUNT; i++) {
        std::memset(m + i, 0, sizeof(CUtensorMap));
        const bool used = vti || i == MM_MU || i == MM_Q || i == MM_RHO || i == MM_IR;
        if (!used) continue;
        const cudaError_t e = encode(m + i, p[i], 2, dim, i < MM_RHO ? halo : own);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_fused(int kind, const ShotDev *shots, const BandRef *bands, int nband, const WinRef *in, int nin,
                         const ModelDev &M, const StepConst &C, int it0, int it1, int flags, float dtg, unsigned *count,
                         int *status, const FluidArgs *fluid, cudaStream_t st)
{
    if (nband + nin <= 0 || it1 <= it0) return cudaSuccess;
    FusedArgs A;
    A.shots = shots;
    A.bands = bands;
    A.in = in;
    A.nband = nband;
    A.nunit = nband + nin;
    A.M = M;
    A.C = C;
    A.it0 = it0;
    A.it1 = it1;
    A.flags = flags;
    A.dtg = dtg;
    A.count = count;
    A.status = status;
    if (fluid) A.W = *fluid;
    const cudaError_t e = model_maps(A.mm, kind, M);
    if (e != cudaSuccess) return e;
    const bool g = (flags & F_GRAD) != 0;
    if (kind == KIND_VTI) return g ? launch_fused_t<true, true, false>(A, st) : launch_fused_t<true, false, false>(A, st);
    if (kind == KIND_AE) return g ? launch_fused_t<false, true, true>(A, st) : launch_fused_t<false, false, true>(A, st);
    return g ? launch_fused_t<false, true, false>(A, st) : launch_fused_t<false, false, false>(A, st);
}

cudaError_t launch_acoustic_loop(const ShotDev *shots, const TileRef *tiles, int ntile, const ModelDev &M, const StepConst &C,
                                 int it0, int it1, int flags, float dtg, unsigned *count, int *status, cudaStream_t st)
{
    if (ntile <= 0 || it1 <= it0) return cudaSuccess;
    const AcousticArgs A = {shots, tiles, ntile, M, C, it0, it1, flags, dtg, count, status};
    if (flags & F_GRAD) return launch_loop(acoustic_steps<true>, A, ntile, sizeof(float) * AcLayout<true>::FLOATS, count, st);
    return launch_loop(acoustic_steps<false>, A, ntile, sizeof(float) * AcLayout<false>::FLOATS, count, st);
}

}  // namespace fwi2d

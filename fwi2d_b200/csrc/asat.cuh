// Acoustic pieces shared by the launch-per-step kernels (acoustic.cuh) and the
// fused time loop (fused.cu): one SAT side at one cell, and the coupling of the
// fluid layer and the elastic grid of the acoustic-elastic propagator.
#pragma once
#include <cuda_runtime.h>
#include "engine.h"
#include "sbp.cuh"
#include "snap.cuh"

namespace fwi2d {

// One SAT side of the acoustic step at one cell (x, z); `side` 0 top,
// 1 bottom, 2 left, 3 right.  U / IR point at the cell inside the tile
// arrays, su / sw are the strides across the side (into the domain), k the
// cell's distance from the side.
__device__ __forceinline__ float asat_cell(float n, int side, int bc, int k, const float *U, int su, const float *IR,
                                           int sw, float p, float K, const StepConst &C)
{
    const bool zside = side < 2;
    const float d = zside ? C.dz : C.dx;
    const float d2 = zside ? C.d2z : C.d2x;
    if (bc == 1) {
        if (k < 4) {
            // the side's boundary sample of this line feeds the first four cells (asat_dirichlet_*)
            const float in = U[-k * su], ir = IR[-k * sw];
            n = (float)((double)n + 1.0 / (double)(kHC[k] * d2) * (double)kSC[k] * (double)ir * (double)in);
        }
        if (k == 0) n = n - IR[0] * U[0] / (C.alpha * kHC[0] * d2);
    } else if (k == 0) {
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < 4; j++) s += kSC[j] * U[j * su];
        const double a = 1.0 / (double)(kHC[0] * d);
        if (bc == 2)
            n = (float)((double)n - a * ((double)(IR[0] * s / d) - (double)p / ((double)(2 * C.dt) * sqrt((double)(K / IR[0])))));
        else
            n = (float)((double)n - a * (double)IR[0] * (double)s / (double)d);
    }
    return n;
}

// Implicit coupling of the fluid potential and the elastic uz at the
// interface (we_op.cpp:2486-2512, the it >= 0 branch) in column ix, after the
// fluid and the elastic part of the step, then the taper of the two interface
// rows.  Every thread of a warp calls it.
// e, w: the elastic and fluid tables of the shot; prev of both interface rows
// (already tapered) is in halo_save.  sign = +1 forward, -1 adjoint.  With
// F_GRAD, the density term of the imaging condition on the interface row,
// which needs the coupled uz (the elastic kernel leaves it out there).
__device__ __forceinline__ void ae_couple_column(const ShotDev &e, const ShotDev &w, int ix, const ModelDev &M,
                                                 const StepConst &C, int it, int flags, float dtg, float Kw, float val0,
                                                 int sign)
{
    if (it >= e.nt - 1) return;
    const long long nxz = (long long)e.nx * e.ldz;
    float *n1 = e.u[it & 1] + nxz;              // next uz, row 0
    float *na = w.u[it & 1] + (w.nz - 1);       // next potential, last fluid row
    float amax = 0.f;   // of the coupled row, which the elastic kernel's maximum has not seen
    if (ix < e.nx) {
        const long long ie = (long long)ix * e.ldz, ia = (long long)ix * w.ldz;
        const float p1 = __ldcg(e.halo_save + ix), pa = __ldcg(w.halo_save + ix);
        const float n1v = __ldcg(n1 + ie), nav = __ldcg(na + ia);
        const float rho = M.p2[(long long)(e.x0 + ix) * M.ldz];
        const float v1 = Kw * val0 * (n1v - p1 + sign * val0 / rho * pa);
        const float v2 = 1 + val0 * val0 * Kw / rho;
        const float a = (nav + sign * v1) / v2;
        const float b = n1v - sign * val0 / rho * (a - pa);
        na[ia] = a * w.tz[w.nz - 1] * w.tx[ix];
        const float a1 = b * e.tz[0] * e.tx[ix];
        n1[ie] = a1;
        amax = fabsf(a1);
        const int tt = e.nt - 1 - (it + 1);
        if ((flags & F_GRAD) && tt % C.sub == 0 && tt / C.sub != 0) {
            // density term at snapshot itf with the coupled next field, as the
            // elastic kernel's (nl_we_op_e::compute_gradients, we_op.cpp:505-562)
            const int itf = tt / C.sub, last = e.nt / C.sub, prec = C.snap_prec;
            const float inv = prec == SNAP_FP32 ? 1.f : 1.f / snap_scale(e.snap_amax, itf);
            const long long o = (long long)itf * e.snap_slot + ie;
            const float f0 = snap_load(e.snap, o, prec, inv), f1 = snap_load(e.snap, o + nxz, prec, inv);
            float fp0 = 0.f, fp1 = 0.f, fm0 = 0.f, fm1 = 0.f;
            if (itf + 1 <= last) {
                const float iv = prec == SNAP_FP32 ? 1.f : 1.f / snap_scale(e.snap_amax, itf + 1);
                const long long op = (long long)(itf + 1) * e.snap_slot + ie;
                fp0 = snap_load(e.snap, op, prec, iv);
                fp1 = snap_load(e.snap, op + nxz, prec, iv);
            }
            {
                const float iv = prec == SNAP_FP32 ? 1.f : 1.f / snap_scale(e.snap_amax, itf - 1);
                const long long om = (long long)(itf - 1) * e.snap_slot + ie;
                fm0 = snap_load(e.snap, om, prec, iv);
                fm1 = snap_load(e.snap, om + nxz, prec, iv);
            }
            const float a0 = __ldcg(e.u[it & 1] + ie);
            const float gw = e.gwt[itf];
            const double wdt = (double)gw * 1.0 / (double)dtg;
            float *g2 = e.grad + 2 * nxz + ie;
            if (itf < last)
                *g2 = (float)((double)__ldcg(g2) + wdt * (double)(a0 * (fp0 - 2 * f0 + fm0) + a1 * (fp1 - 2 * f1 + fm1)));
            else
                *g2 = (float)((double)__ldcg(g2) + wdt * (double)(a0 * (-f0 + fm0) + a1 * (-f1 + fm1)));
        }
    }
    if ((flags & F_AMAX) && (it + 1) % C.sub == 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        if ((threadIdx.x & 31) == 0 && amax > 0.f) atomicMax(e.snap_amax + (it + 1) / C.sub, __float_as_uint(amax));
    }
}

}  // namespace fwi2d

// Kernel bodies shared by the per-precision translation units.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <type_traits>

#include "geopotential.cuh"
#include "nrlmsise00.cuh"
#include "propagate.cuh"

namespace phop {


// ---- RKF78 tableau (parm/integrate/rk/coefs/tableau.h:24-48) ----------------------------
__host__ __device__ constexpr double rkA(int s, int j) {
    // s = stage - 1 (row), j = column; rows list the nonzero Fehlberg coefficients
    return s == 0 ? (j == 0 ? 2. / 27 : 0)
         : s == 1 ? (j == 0 ? 1. / 36 : j == 1 ? 1. / 12 : 0)
         : s == 2 ? (j == 0 ? 1. / 24 : j == 2 ? 1. / 8 : 0)
         : s == 3 ? (j == 0 ? 5. / 12 : j == 2 ? -25. / 16 : j == 3 ? 25. / 16 : 0)
         : s == 4 ? (j == 0 ? 1. / 20 : j == 3 ? 1. / 4 : j == 4 ? 1. / 5 : 0)
         : s == 5 ? (j == 0 ? -25. / 108 : j == 3 ? 125. / 108 : j == 4 ? -65. / 27 : j == 5 ? 125. / 54 : 0)
         : s == 6 ? (j == 0 ? 31. / 300 : j == 4 ? 61. / 225 : j == 5 ? -2. / 9 : j == 6 ? 13. / 900 : 0)
         : s == 7 ? (j == 0 ? 2.0 : j == 3 ? -53. / 6 : j == 4 ? 704. / 45 : j == 5 ? -107. / 9
                    : j == 6 ? 67. / 90 : j == 7 ? 3.0 : 0)
         : s == 8 ? (j == 0 ? -91. / 108 : j == 3 ? 23. / 108 : j == 4 ? -976. / 135 : j == 5 ? 311. / 54
                    : j == 6 ? -19. / 60 : j == 7 ? 17. / 6 : j == 8 ? -1. / 12 : 0)
         : s == 9 ? (j == 0 ? 2383. / 4100 : j == 3 ? -341. / 164 : j == 4 ? 4496. / 1025 : j == 5 ? -301. / 82
                    : j == 6 ? 2133. / 4100 : j == 7 ? 45. / 82 : j == 8 ? 45. / 164 : j == 9 ? 18. / 41 : 0)
         : s == 10 ? (j == 0 ? 3. / 205 : j == 5 ? -6. / 41 : j == 6 ? -3. / 205 : j == 7 ? -3. / 41
                     : j == 8 ? 3. / 41 : j == 9 ? 6. / 41 : 0)
         : s == 11 ? (j == 0 ? -1777. / 4100 : j == 3 ? -341. / 164 : j == 4 ? 4496. / 1025 : j == 5 ? -289. / 82
                     : j == 6 ? 2193. / 4100 : j == 7 ? 51. / 82 : j == 8 ? 33. / 164 : j == 9 ? 12. / 41
                     : j == 11 ? 1.0 : 0)
         : 0;
}
__host__ __device__ constexpr double rkC(int s) {
    return s == 0 ? 2. / 27 : s == 1 ? 1. / 9 : s == 2 ? 1. / 6 : s == 3 ? 5. / 12 : s == 4 ? 1. / 2
         : s == 5 ? 5. / 6 : s == 6 ? 1. / 6 : s == 7 ? 2. / 3 : s == 8 ? 1. / 3 : s == 9 ? 1.0
         : s == 10 ? 0 : 1.0;
}
__host__ __device__ constexpr double rkB(int s) {
    return s == 5 ? 34. / 105 : s == 6 ? 9. / 35 : s == 7 ? 9. / 35 : s == 8 ? 9. / 280 : s == 9 ? 9. / 280
         : s == 11 ? 41. / 840 : s == 12 ? 41. / 840 : 0;
}

// ---- RK stages on accelerations alone -------------------------------------------------------
// The right-hand side is y'' = f(t, y, y'), so the position rows of the stage
// sums are sums of the velocity rows' own sums: with k_j the accelerations,
//     v_s = v + dt sum_j a_sj k_j
//     y_s = y + dt c_s v + dt^2 sum_j (A A)_sj k_j
// and the same for the update with b and b A.  Only accelerations are kept:
// ten slots of three doubles an object, against thirteen stages of six
// components.  Stage 10 (c = 1) enters neither another stage nor the
// 8th-order update (it serves the 7th-order error estimate, which a fixed
// step does not form), so it is not evaluated; stage 11 takes the slot of
// stage 1, whose last reader is stage 4.  rkAA and rkBA are the exact
// rational products.  At one lane per object the 624 bytes of stage
// derivatives an object left 128 threads a CTA beside the degree-70 tile; 240
// bytes leave room for all 256: 200,000 uneven objects x 8 steps FP64 86.6 ->
// 66.3 ms, 10^6 x 4 split 126 -> 110 ms, 10^4 LEO x 20 FP64 16.2 -> 14.9 ms.
__host__ __device__ constexpr double rkAA(int s, int j) {
    return s == 2 ? (j == 0 ? 1. / 162 : 0)
         : s == 3 ? (j == 0 ? 1. / 288 : j == 1 ? 1. / 96 : 0)
         : s == 4 ? (j == 0 ? 25. / 1152 : j == 1 ? -25. / 192 : j == 2 ? 25. / 128 : 0)
         : s == 5 ? (j == 0 ? 3. / 32 : j == 2 ? -9. / 32 : j == 3 ? 5. / 16 : 0)
         : s == 6 ? (j == 0 ? -725. / 864 : j == 2 ? 125. / 32 : j == 3 ? -1375. / 432 : j == 4 ? 25. / 54 : 0)
         : s == 7 ? (j == 0 ? 383. / 3888 : j == 2 ? -61. / 144 : j == 3 ? 187. / 486 : j == 4 ? -77. / 972
                    : j == 5 ? 65. / 1944 : 0)
         : s == 8 ? (j == 0 ? 553427. / 97200 : j == 2 ? -3679. / 144 : j == 3 ? 43417. / 1944
                    : j == 4 ? -40783. / 12150 : j == 5 ? 1027. / 972 : j == 6 ? 13. / 300 : 0)
         : s == 9 ? (j == 0 ? -163043. / 64800 : j == 2 ? 1087. / 96 : j == 3 ? -12295. / 1296
                    : j == 4 ? 11167. / 8100 : j == 5 ? -241. / 648 : j == 6 ? -19. / 900 : j == 7 ? -1. / 4 : 0)
         : s == 11 ? (j == 0 ? 71. / 6150 : j == 3 ? -329. / 492 : j == 4 ? 224. / 3075 : j == 5 ? -11. / 246
                     : j == 6 ? 29. / 4100 : j == 7 ? 26. / 41 : j == 8 ? -1. / 82 : 0)
         : s == 12 ? (j == 0 ? 54963. / 32800 : j == 2 ? -9333. / 1312 : j == 3 ? 3199. / 656
                     : j == 4 ? -3247. / 4100 : j == 5 ? 81. / 328 : j == 6 ? 211. / 4100 : j == 7 ? 223. / 164
                     : j == 8 ? 2. / 41 : j == 9 ? 6. / 41 : 0)
         : 0;
}
__host__ __device__ constexpr double rkBA(int j) {
    return j == 5 ? 17. / 105 : j == 6 ? 3. / 70 : j == 7 ? 3. / 14 : j == 8 ? 3. / 280 : j == 9 ? 3. / 140
         : j == 11 ? 41. / 840 : 0;
}
__host__ __device__ constexpr int rkSlot(int s) { return s == 11 ? 1 : s; }

// A lane owns AXES coordinate axes (position and velocity): all three at one
// lane per object; axes j and 2 at two lanes (both lanes carry axis 2); axis
// j % 3 at four and more.  The accelerations of the stages lie in shared
// memory, [slot][axis][object of the CTA].
template <int L>
struct Axes {
    static constexpr int N = L == 1 ? 3 : L == 2 ? 2 : 1;
    static __device__ __forceinline__ int axis(int j, int i) {
        return L == 1 ? i : L == 2 ? (i == 0 ? j : 2) : j % 3;
    }
    // the lane that writes axis(j, i) to memory
    static __device__ __forceinline__ bool writes(int j, int i) {
        return L == 1 ? true : L == 2 ? (i == 0 || j == 0) : j < 3;
    }
    // lane and place of axis a
    static __host__ __device__ constexpr int lane(int a) { return L == 1 ? 0 : L == 2 ? (a == 2 ? 0 : a) : a; }
    static __host__ __device__ constexpr int place(int a) { return L == 1 ? a : L == 2 ? (a == 2 ? 1 : 0) : 0; }
};

struct StageStore {
    double* base;  // this object's first slot
    int stride;    // objects of the CTA
    __device__ __forceinline__ double& at(int slot, int axis) const { return base[(slot * 3 + axis) * stride]; }
};

// position and velocity of the lane's axes at stage S
template <int L, int S>
static __device__ __forceinline__ void stageState(const double (&y)[Axes<L>::N], const double (&v)[Axes<L>::N],
                                                  const StageStore& k, int j, double dt, double (&ys)[Axes<L>::N],
                                                  double (&vs)[Axes<L>::N]) {
    const double dt2 = dt * dt;
#pragma unroll
    for (int i = 0; i < Axes<L>::N; ++i) {
        const int axis = Axes<L>::axis(j, i);
        double sv = 0.0, sy = 0.0;
#pragma unroll
        for (int l = 0; l < S; ++l) {
            if (rkA(S - 1, l) != 0.0 || rkAA(S, l) != 0.0) {
                const double kl = k.at(rkSlot(l), axis);
                if (rkA(S - 1, l) != 0.0) sv = fma(rkA(S - 1, l), kl, sv);
                if (rkAA(S, l) != 0.0) sy = fma(rkAA(S, l), kl, sy);
            }
        }
        ys[i] = fma(dt2, sy, fma(dt * rkC(S - 1), v[i], y[i]));
        vs[i] = fma(dt, sv, v[i]);
    }
}

// the 8th-order update of the lane's axes; acc is stage 12's acceleration
template <int L>
static __device__ __forceinline__ void finalUpdate(double (&y)[Axes<L>::N], double (&v)[Axes<L>::N],
                                                   const StageStore& k, int j, double dt, const double acc[3],
                                                   bool apply) {
#pragma unroll
    for (int i = 0; i < Axes<L>::N; ++i) {
        const int axis = Axes<L>::axis(j, i);
        double sv = 0.0, sy = 0.0;
#pragma unroll
        for (int l = 5; l < 12; ++l)
            if (rkB(l) != 0.0) {
                const double kl = k.at(rkSlot(l), axis);
                sv = fma(rkB(l), kl, sv);
                sy = fma(rkBA(l), kl, sy);
            }
        sv = fma(rkB(12), axis == 0 ? acc[0] : axis == 1 ? acc[1] : acc[2], sv);
        if (apply) {
            y[i] = fma(dt, fma(dt, sy, v[i]), y[i]);
            v[i] = fma(dt, sv, v[i]);
        }
    }
}

// ---- epoch records as the force model reads them -----------------------------------------
// A shared-grid batch reads the precomputed record of its (step, stage) in
// place.  A per-object-time batch interpolates each field where the force
// model reads it (4-point Lagrange in the batch's record grid, weights
// depending on the epoch alone), so no record is copied into the thread's
// local memory.
struct RecordRef {
    const EpochRecord* r;
    __device__ __forceinline__ double R(int i) const { return r->R[i]; }
    __device__ __forceinline__ double W(int i) const { return r->w[i]; }
    __device__ __forceinline__ double body(int b, int i) const { return r->body[b][i]; }
    __device__ __forceinline__ double indirect(int i) const { return r->indirect[i]; }
    __device__ __forceinline__ double dC(int k) const { return r->dC[k]; }
    __device__ __forceinline__ double dS(int k) const { return r->dS[k]; }
    __device__ __forceinline__ double pole(int k, int i) const { return r->pole[k][i]; }
    __device__ __forceinline__ double poleW(int k, int i) const { return r->poleW[k][i]; }
    __device__ __forceinline__ double poleV(int k, int i) const { return r->poleV[k][i]; }
    __device__ __forceinline__ double SR(int i) const { return r->fieldR[i]; }
    // NRLMSISE-00 time inputs; valid = -1 (evaluate at the epoch in `sec`
    // when an object below the cut-off needs them) when the record has none
    __device__ __forceinline__ NrlTime nrlDeferred() const {
        NrlTime t{r->nrlSec, r->nrlGast, r->nrlBlock, r->nrlValid};
        if (t.valid < 0) t.sec = r->et;
        return t;
    }
};

struct RecordInterp {
    // value pairs of the stencil's records i0, i0 + 1 (field f at g[f]); those
    // of records i0 + 2, i0 + 3 follow 2 kInterpFields pairs later
    const double2* g;
    double w0, w1, w2, w3;
    double et;        // the stage epoch (TDB s past J2000)
    // explicit roundings: every copy of this code gives the same bits
    __device__ __forceinline__ double at(int off) const {
        const double2 x = g[off], y = g[2 * kInterpFields + off];
        return __fma_rn(w3, y.y, __fma_rn(w2, y.x, __fma_rn(w1, x.y, __dmul_rn(w0, x.x))));
    }
    __device__ __forceinline__ double R(int i) const { return at((int)(offsetof(EpochRecord, R) / 8) + i); }
    __device__ __forceinline__ double W(int i) const { return at((int)(offsetof(EpochRecord, w) / 8) + i); }
    __device__ __forceinline__ double body(int b, int i) const {
        return at((int)(offsetof(EpochRecord, body) / 8) + 3 * b + i);
    }
    __device__ __forceinline__ double indirect(int i) const {
        return at((int)(offsetof(EpochRecord, indirect) / 8) + i);
    }
    __device__ __forceinline__ double dC(int k) const { return at((int)(offsetof(EpochRecord, dC) / 8) + k); }
    __device__ __forceinline__ double dS(int k) const { return at((int)(offsetof(EpochRecord, dS) / 8) + k); }
    __device__ __forceinline__ double pole(int k, int i) const {
        return at((int)(offsetof(EpochRecord, pole) / 8) + 3 * k + i);
    }
    __device__ __forceinline__ double poleW(int k, int i) const {
        return at((int)(offsetof(EpochRecord, poleW) / 8) + 3 * k + i);
    }
    __device__ __forceinline__ double poleV(int k, int i) const {
        return at((int)(offsetof(EpochRecord, poleV) / 8) + 3 * k + i);
    }
    __device__ __forceinline__ double SR(int i) const { return at((int)(offsetof(EpochRecord, fieldR) / 8) + i); }
    // NRLMSISE-00 time inputs: evaluated exactly at the stage epoch by the
    // drag model, only for objects below the density cut-off
    __device__ __forceinline__ NrlTime nrlDeferred() const { return NrlTime{et, 0.0, 0, -1}; }
};

// body-fixed (ITRF) components of an inertial vector, and back
template <class Rec>
static __device__ __forceinline__ void toBody(const Rec& r, const double v[3], double out[3]) {
    out[0] = r.R(0) * v[0] + r.R(1) * v[1] + r.R(2) * v[2];
    out[1] = r.R(3) * v[0] + r.R(4) * v[1] + r.R(5) * v[2];
    out[2] = r.R(6) * v[0] + r.R(7) * v[1] + r.R(8) * v[2];
}
template <class Rec>
static __device__ __forceinline__ void fromBody(const Rec& r, const double a[3], double out[3]) {
    out[0] = r.R(0) * a[0] + r.R(3) * a[1] + r.R(6) * a[2];
    out[1] = r.R(1) * a[0] + r.R(4) * a[1] + r.R(7) * a[2];
    out[2] = r.R(2) * a[0] + r.R(5) * a[1] + r.R(8) * a[2];
}

// ---- the remaining forces ------------------------------------------------------------------
static __device__ __forceinline__ double shadowFactor(const double rS[3], const double rB[3], double RSun, double RBody) {
    const double s2 = rS[0] * rS[0] + rS[1] * rS[1] + rS[2] * rS[2];
    const double b2 = rB[0] * rB[0] + rB[1] * rB[1] + rB[2] * rB[2];
    const double sb = rS[0] * rB[0] + rS[1] * rB[1] + rS[2] * rB[2];
    const double iS = rsqrt(s2), iB = rsqrt(b2);
    if (b2 <= RBody * RBody) return 0.0;
    {
        // clear full sunlight (c > a + b) or full shadow of a body larger
        // than the Sun's disc (c < b - a), decided on cosines without the
        // inverse trigonometric functions; within 1e-9 of either boundary
        // the angles below decide, as the reference's evaluation does
        const double sa = fmin(fmax(RSun * iS, 0.0), 1.0), sbd = fmin(fmax(RBody * iB, 0.0), 1.0);
        const double ca = sqrt(1.0 - sa * sa), cb = sqrt(1.0 - sbd * sbd);
        const double cc = fmin(fmax(sb * iS * iB, -1.0), 1.0);
        if (cc < ca * cb - sa * sbd - 1e-9) return 1.0;
        if (sbd > sa && cc > ca * cb + sa * sbd + 1e-9) return 0.0;
    }
    const double a = asin(fmin(fmax(RSun * iS, 0.0), 1.0));
    const double b = asin(fmin(fmax(RBody * iB, 0.0), 1.0));
    const double c = acos(fmin(fmax(sb * iS * iB, -1.0), 1.0));
    if (c >= a + b) return 1.0;
    if (c <= fabs(b - a)) return b >= a ? 0.0 : 1.0 - (b * b) / (a * a);
    const double a2 = a * a, bb = b * b, c2 = c * c;
    const double x = (c2 + a2 - bb) / (2.0 * c);
    const double yv = sqrt(fmax(a2 - x * x, 0.0));
    const double al = acos(fmin(fmax(x / a, -1.0), 1.0));
    const double be = acos(fmin(fmax((c - x) / b, -1.0), 1.0));
    return 1.0 - (a2 * al + bb * be - c * yv) / (a2 * 3.14159265358979323846);
}

// NRLMSISE-00 density (kg/km^3) at ITRF position f; the L lanes of a group
// share the globe7 tables of the model and all return the same value.
template <int L>
static __device__ __forceinline__ double nrlDensityBody(const DevEnv& e, NrlTime t, const double f[3]);

// Out of line for eight and sixteen lanes, where the caller's live state is
// small enough that the call's register saves cost less than the larger
// inlined kernel; inline for one to four lanes (measured both ways).
template <int L>
static __device__ __noinline__ double nrlDensityCall(const DevEnv& e, NrlTime t, const double f[3]) {
    return nrlDensityBody<L>(e, t, f);
}
// FP64 in both precision forms: an FP32 per-object model (the split form's
// option at one time) was slower and moved 500 km objects by more than 1 cm
// in 24 h.
template <int L>
static __device__ __forceinline__ double nrlDensity(const DevEnv& e, NrlTime t, const double f[3]) {
    if constexpr (L <= 4) return nrlDensityBody<L>(e, t, f);
    else return nrlDensityCall<L>(e, t, f);
}

template <int L>
static __device__ __forceinline__ double nrlDensityBody(const DevEnv& e, NrlTime t, const double f[3]) {
    // geodetic latitude / longitude / altitude (Nrlmsise00.cu:243-266)
    const double rho2 = f[0] * f[0] + f[1] * f[1], r2 = rho2 + f[2] * f[2];
    if (!(r2 > 0.0)) return NAN;
    const double radius = e.earthRadius;
    // an oblate ellipsoid lies inside the sphere of its equatorial radius:
    // above the cut-off from there is above it everywhere
    const bool oblate = e.flattening >= 0.0 && e.flattening < 1.0;
    const double clear = radius + e.nrlHcutoff;
    if (oblate && e.nrlHcutoff >= 0.0 && r2 > clear * clear && r2 < 1e30) return 0.0;
    const double e2 = e.flattening * (2.0 - e.flattening);
    const double rho = sqrt(rho2);
    double dz = e2 * f[2], zdz, nn = radius, nh = 0.0;
    if (oblate) {
        // start from Bowring's latitude (Survey Review 23(181), 1976), off by
        // less than 1e-11 rad in orbit, so that the fixed point below ends
        // after one pass instead of five (with the angle rotations below, a
        // density above 450 km at sixteen lanes, one warp: 12.5 -> 11.3
        // thousand cycles)
        const double b = radius * (1.0 - e.flattening);
        const double za = f[2] * radius, pb = rho * b;
        const double q = rsqrt(za * za + pb * pb);
        const double su = za * q, cu = pb * q;
        const double num = f[2] + e2 / (1.0 - e2) * b * (su * su * su), den = rho - e2 * radius * (cu * cu * cu);
        const double sp = num * rsqrt(num * num + den * den);
        dz = e2 * sp * radius * rsqrt(1.0 - e2 * sp * sp);
    }
    for (int it = 0; it < 20; ++it) {
        zdz = f[2] + dz;
        const double sp = zdz * rsqrt(rho2 + zdz * zdz);
        nn = radius * rsqrt(1.0 - e2 * sp * sp);
        const double next = nn * e2 * sp;
        if (fabs(dz - next) < 1.0e-12 * radius) {
            dz = next;
            break;
        }
        dz = next;
    }
    zdz = f[2] + dz;
    nh = sqrt(rho2 + zdz * zdz);
    const double lon = atan2(f[1], f[0]);
    const double lat = atan2(zdz, rho);
    const double alt = nh - nn;
    if (!(isfinite(lat) && isfinite(lon) && isfinite(alt))) return NAN;
    if (alt > e.nrlHcutoff) return 0.0;
    if (t.valid < 0) t = nrlTime(e, t.sec);  // deferred: `sec` holds the stage epoch (TDB s past J2000)
    if (!t.valid) return NAN;
    const double kRad = 57.2957795130823208768;
    // hours in [0, 24): the sum of two such angles is out by one turn at most
    const double hours = t.gast + lon * kRad / 15.0;
    const double lst = hours >= 0.0 && hours < 24.0     ? hours
                       : hours >= 24.0 && hours < 48.0 ? hours - 24.0
                                                       : wrapHours(hours);
    // sines and cosines of the model's latitude and longitude angles (degrees
    // by its own rounded factor) from the coordinates
    const double inh = 1.0 / nh, irho = rho > 0.0 ? 1.0 / rho : 0.0;
    nrlf::Angles<double> ang;
    ang.latitude(zdz * inh, rho * inh, lat);
    ang.longitude(rho > 0.0 ? f[1] * irho : 0.0, rho > 0.0 ? f[0] * irho : 1.0, lon);
    const int lane = (int)(threadIdx.x & 31);
    nrlf::Fast<double> model(e.nrlBlocks[t.block], t.sec);
    const double rhoSi = model.template density<L>(lat * kRad, lon * kRad, alt, lst, ang, lane % L, lane - lane % L);
    if (!isfinite(rhoSi) || rhoSi < 0.0) return NAN;
    return (rhoSi * 1.0e9) * e.nrlDensityScale;
}

// Geodetic altitude about the polar axis `pole` (atmosphere/Geodetic.h:40-75);
// the fixed-point iteration converges quadratically, bounded here.
static __device__ __forceinline__ double geodeticHeight(const double r[3], const double pole[3], double Req,
                                                        double flattening) {
    const double r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
    if (flattening == 0.0) return sqrt(r2) - Req;
    const double z = r[0] * pole[0] + r[1] * pole[1] + r[2] * pole[2];
    const double xy = r2 - z * z;
    const double flatsq = (2.0 - flattening) * flattening;
    double d0 = 0.0, d = 1e10, sfq = 0.0, zd = z;
    for (int it = 0; it < 64 && fabs(d - d0) > 1e-9; ++it) {
        d0 = d;
        const double z2 = zd * zd;
        sfq = z2 / (xy + z2);
        d = Req * flatsq * sqrt(sfq / (1.0 - flatsq * sfq));
        zd = z + copysign(d, z);
    }
    return sqrt(xy + zd * zd) - Req / sqrt(1.0 - flatsq * sfq);
}

// Tide potential alone (solid + ocean coefficient deltas of the epoch, degree
// <= 6, the tide model's GM and radius), for an Earth without a gravity field
// file: the deltas otherwise join the field's low-degree block.  The body-
// frame gradient of sum_nm (mu/r)(R/r)^n P_nm (dC cos m lon + dS sin m lon)
// in geocentric latitude/longitude, as the reference's Earth corrections
// evaluate it (hpop_compat/HpopCorrections.h:336-367); fully normalised
// Legendre functions by the column recurrences and their latitude
// derivatives in closed form (the reference recurses them alongside,
// HpopCorrections.h:121-145).
template <class Rec>
static __device__ __noinline__ void tideAloneAccel(const Rec r, const double pos[3], double acc[3]) {
    double b[3];
    toBody(r, pos, b);
    const double x = b[0], y = b[1], z = b[2];
    const double mu = tidefield::kMuEarth * 1e-9, Re = tidefield::kRadius * 1e-3;  // km^3/s^2, km
    const double xy2 = x * x + y * y, xy = sqrt(xy2);
    const double d = sqrt(xy2 + z * z);
    const double sphi = z / d, cphi = xy / d, tphi = z / xy;
    const double cl = x / xy, sl = y / xy;
    double p[7][7], dp[7][7];
    // column recurrences: P_mm from P_{m-1,m-1}, then upward in n
    p[0][0] = 1.0;
    for (int m = 0; m <= 6; ++m) {
        if (m > 0) p[m][m] = sqrt((2.0 * m + 1.0) / (m == 1 ? 1.0 : 2.0 * m)) * cphi * p[m - 1][m - 1];
        if (m < 6) p[m + 1][m] = sqrt(2.0 * m + 3.0) * sphi * p[m][m];
        for (int n = m + 2; n <= 6; ++n) {
            const double nn = (double)n, mm = (double)m;
            const double a = sqrt((4.0 * nn * nn - 1.0) / (nn * nn - mm * mm));
            const double b = sqrt((2.0 * nn + 1.0) * (nn - 1.0 - mm) * (nn - 1.0 + mm) / ((2.0 * nn - 3.0) * (nn * nn - mm * mm)));
            p[n][m] = a * sphi * p[n - 1][m] - b * p[n - 2][m];
        }
    }
    // d/dphi P_nm = k_nm P_{n,m+1} - m tan(phi) P_nm, k_n0 = sqrt(n(n+1)/2), k_nm = sqrt((n-m)(n+m+1))
    for (int n = 0; n <= 6; ++n)
        for (int m = 0; m <= n; ++m) {
            const double up = m < n ? p[n][m + 1] : 0.0;
            const double k = m == 0 ? sqrt(0.5 * n * (n + 1.0)) : sqrt((double)(n - m) * (n + m + 1.0));
            dp[n][m] = k * up - (double)m * tphi * p[n][m];
        }
    double cm[7], sm[7];
    cm[0] = 1.0;
    sm[0] = 0.0;
    for (int m = 1; m <= 6; ++m) {
        cm[m] = cl * cm[m - 1] - sl * sm[m - 1];
        sm[m] = sl * cm[m - 1] + cl * sm[m - 1];
    }
    double dUdr = 0.0, dUdlat = 0.0, dUdlon = 0.0, power = 1.0;
    const double ratio = Re / d;
    for (int n = 0; n <= 6; ++n) {
        double q1 = 0.0, q2 = 0.0, q3 = 0.0;
        for (int m = 0; m <= n; ++m) {
            const int ti = n * (n + 1) / 2 + m;
            const double c = r.dC(ti), s = r.dS(ti);
            const double v = c * cm[m] + s * sm[m];
            q1 += p[n][m] * v;
            q2 += dp[n][m] * v;
            q3 += (double)m * p[n][m] * (s * cm[m] - c * sm[m]);
        }
        dUdr += q1 * (-mu / (d * d)) * power * (n + 1.0);
        dUdlat += q2 * (mu / d) * power;
        dUdlon += q3 * (mu / d) * power;
        power *= ratio;
    }
    const double q = dUdr / d - z / (d * d * xy) * dUdlat;
    const double bf0 = q * x - (dUdlon / xy2) * y, bf1 = q * y + (dUdlon / xy2) * x;
    const double bf2 = dUdr / d * z + xy / (d * d) * dUdlat;
    const double bf[3] = {bf0, bf1, bf2};
    double a[3];
    fromBody(r, bf, a);
    acc[0] += a[0];
    acc[1] += a[1];
    acc[2] += a[2];
}

// ---- drag on a warp of its own -----------------------------------------------------------------
// A small batch leaves the GPU all but empty, and its time is the latency of
// one warp's force model: at sixteen lanes an evaluation below 450 km is some
// 60 thousand cycles, 25 of them NRLMSISE-00, whose inputs are known at the
// start.  So warps work in pairs: the main warp posts the body-fixed positions
// and time inputs of its objects, its partner evaluates the densities while
// the main warp does everything else, and the main warp picks them up.  The
// pair meets at two named barriers an evaluation (post: main arrives, partner
// waits; reply: partner arrives, main waits), so either side's writes are
// ordered before the other's reads, and neither overwrites what the other may
// still read.  Kernel, ten steps at degree 70: 33
// objects 3.77 -> 2.04 ms, 1,000 4.28 -> 2.12, 4,000 4.81 -> 3.34.
struct Duo {
    DuoMail* mail;  // of the pair's objects, 32 / L
    int* quit;
    int barrier;    // the post barrier; the reply barrier is the next
};
// Both forms are aligned: all lanes of a warp execute them together, which the
// force model's per-lane branches (shadow, spheres of influence) before the
// reply would otherwise leave to the compiler.  The warp's synchronisation
// also orders its lanes' accesses to the mail.
static __device__ __forceinline__ void duoArrive(int id) {
    __syncwarp();
    asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory");
}
static __device__ __forceinline__ void duoSync(int id) {
    __syncwarp();
    asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
}

// the partner's loop
template <int L>
static __device__ __forceinline__ void duoPartner(const DevEnv& e, const Duo& duo) {
    const int lane = (int)(threadIdx.x & 31);
    DuoMail& m = duo.mail[lane / L];
    while (true) {
        duoSync(duo.barrier);
        if (*(volatile int*)duo.quit) return;
        const double f[3] = {m.f[0], m.f[1], m.f[2]};
        const double rho = nrlDensity<L>(e, NrlTime{m.sec, m.gast, m.block, m.valid}, f);
        if (lane % L == 0) m.rho = rho;
        duoArrive(duo.barrier + 1);
    }
}

// full right-hand side acceleration (km/s^2); every lane of the group calls it.
// PAIR: two lane groups share their columns (a separate kernel instantiation,
// so the one-object-per-lane kernel keeps its own register allocation).
// NRL: with the NRLMSISE-00 model; DUO: its densities from the partner warp.
template <int L, typename T, bool PAIR, TileRead MODE, bool NRL, bool DUO, class Rec>
static __device__ __forceinline__ void accelerations(const StepParams& p, const TileRef& tile,
                                              TileStream<(PAIR ? 2 : 1) * L>& stream, const Duo& duo, const Rec& r, const double pos[3], const double vel[3],
                                              double bc, double ams, double acc[3]) {
    const DevEnv& e = p.env;
    // read first, used last: the trip to the record overlaps the rest
    double ax = r.indirect(0), ay = r.indirect(1), az = r.indirect(2);
    if constexpr (DUO) {
        double f[3];
        toBody(r, pos, f);
        const int lane = (int)(threadIdx.x & 31);
        if (lane % L == 0) {
            DuoMail& m = duo.mail[lane / L];
            const NrlTime t = r.nrlDeferred();
            for (int k = 0; k < 3; ++k) m.f[k] = f[k];
            m.sec = t.sec;
            m.gast = t.gast;
            m.block = t.block;
            m.valid = t.valid;
        }
        duoArrive(duo.barrier);
    }
    for (int bi = 0; bi < e.nbodies; ++bi) {
        const int fl = e.bodyFlags[bi];
        const bool isEarth = (bi == e.earthIndex);
        // the body-fixed position (field, J2 and NRLMSISE-00 terms) and the
        // body's position (direct attraction and radiation pressure), each
        // read from the record once
        double fb[3] = {0.0, 0.0, 0.0}, rb[3] = {0.0, 0.0, 0.0};
        if (isEarth && ((fl & (kShape | kOblateness)) || (NRL && (fl & kAtmosphere) && e.hasNrl))) toBody(r, pos, fb);
        if (((fl & (kGravity | kAtmosphere)) && !isEarth) || (fl & kRadiation)) {
            rb[0] = r.body(bi, 0);
            rb[1] = r.body(bi, 1);
            rb[2] = r.body(bi, 2);
        }
        if (fl & kGravity) {
            const double gm = e.bodyGm[bi];
            if (isEarth) {
                const double rr = sqrt(pos[0] * pos[0] + pos[1] * pos[1] + pos[2] * pos[2]);
                const double f = -gm * (1.0 / (rr * rr * rr));
                ax += f * pos[0];
                ay += f * pos[1];
                az += f * pos[2];
            } else {
                // direct part per object; the indirect part (epoch-only) is
                // the record's sum, added after the loop
                const double d0 = pos[0] - rb[0], d1 = pos[1] - rb[1], d2 = pos[2] - rb[2];
                const double ird = rsqrt(d0 * d0 + d1 * d1 + d2 * d2);
                const double f1 = -gm * (ird * ird * ird);
                ax += f1 * d0;
                ay += f1 * d1;
                az += f1 * d2;
            }
        }
        if (fl & kShape) {
            // body-fixed position: the Earth's frame, or the field body's
            // own (IAU) frame about its position
            double bx = fb[0], by = fb[1], bz = fb[2];
            if (!isEarth) {
                const double d0 = pos[0] - rb[0], d1 = pos[1] - rb[1], d2 = pos[2] - rb[2];
                bx = r.SR(0) * d0 + r.SR(1) * d1 + r.SR(2) * d2;
                by = r.SR(3) * d0 + r.SR(4) * d1 + r.SR(5) * d2;
                bz = r.SR(6) * d0 + r.SR(7) * d1 + r.SR(8) * d2;
            }
            double a[3];
            // split precision with a floor: objects below the split radius
            // keep every row in FP64 (from the FP64 tile in global memory)
            if (!PAIR && sizeof(T) == 4 && p.splitRadius > 0.0
                && bx * bx + by * by + bz * bz < p.splitRadius * p.splitRadius) {
                TileStream<L> none;
                fieldAccel<L, 1, double, TileRead::kGeneric>(p, TileRef{p.tile64, p.nblocks64, 0}, none, r, bx, by, bz, a);
            } else {
                fieldAccel<L, PAIR ? 2 : 1, T, MODE>(p, tile, stream, r, bx, by, bz, a);
            }
            double ai[3];
            if (isEarth) {
                fromBody(r, a, ai);
            } else {
                ai[0] = r.SR(0) * a[0] + r.SR(3) * a[1] + r.SR(6) * a[2];
                ai[1] = r.SR(1) * a[0] + r.SR(4) * a[1] + r.SR(7) * a[2];
                ai[2] = r.SR(2) * a[0] + r.SR(5) * a[1] + r.SR(8) * a[2];
            }
            ax += ai[0];
            ay += ai[1];
            az += ai[2];
        }
        if ((fl & kOblateness) && !(fl & kShape) && !isEarth) {
            // J2 model of another body (J2.h:17-33,63-78, PrivateAccelerations.h:88-97):
            // position relative to the body, inside its sphere of influence;
            // the model is axisymmetric, so the body frame enters through its
            // polar axis u alone: a = c (d (1 - 5 z^2 / r^2) + 2 z u), z = u . d
            const double d0 = pos[0] - rb[0], d1 = pos[1] - rb[1], d2 = pos[2] - rb[2];
            const double rr2 = d0 * d0 + d1 * d1 + d2 * d2;
            const int slot = e.poleSlot[bi];
            if (slot >= 0 && rr2 <= e.bodySoi[bi] * e.bodySoi[bi]) {
                const double u0 = r.pole(slot, 0), u1 = r.pole(slot, 1), u2 = r.pole(slot, 2);
                const double invr = rsqrt(rr2);
                const double invr2 = invr * invr;
                const double z = u0 * d0 + u1 * d1 + u2 * d2;
                const double base = 1.0 - 5.0 * (z * z) * invr2;
                const double c = -1.5 * e.bodyGmConst[bi] * e.bodyJ2[bi] * (invr2 * invr2 * invr) * e.bodyRadius[bi]
                                 * e.bodyRadius[bi];
                ax += c * (d0 * base + 2.0 * z * u0);
                ay += c * (d1 * base + 2.0 * z * u1);
                az += c * (d2 * base + 2.0 * z * u2);
            }
        }
        if ((fl & kOblateness) && !(fl & kShape) && isEarth) {
            // J2 model in the body frame (J2.h:17-33,63-78), inside the sphere of influence
            const double rr = sqrt(pos[0] * pos[0] + pos[1] * pos[1] + pos[2] * pos[2]);
            if (rr <= e.bodySoi[bi]) {
                const double bx = fb[0], by = fb[1], bz = fb[2];
                const double invr = 1.0 / sqrt(bx * bx + by * by + bz * bz);
                const double invr2 = invr * invr;
                const double invr5 = invr2 * invr2 * invr;
                const double base = 1.0 - 5.0 * (bz * bz) * invr2;
                const double c = -1.5 * e.bodyGmConst[bi] * e.bodyJ2[bi] * invr5 * e.bodyRadius[bi] * e.bodyRadius[bi];
                const double aj[3] = {c * bx * base, c * by * base, c * bz * (base + 2.0)};
                double ai[3];
                fromBody(r, aj, ai);
                ax += ai[0];
                ay += ai[1];
                az += ai[2];
            }
        }
        if (fl & kRadiation) {
            const double dp[3] = {pos[0] - rb[0], pos[1] - rb[1], pos[2] - rb[2]};
            const double ird = rsqrt(dp[0] * dp[0] + dp[1] * dp[1] + dp[2] * dp[2]);
            double occ = 1.0;
            if (e.anyOcculter) {
                for (int oj = 0; oj < e.nbodies; ++oj) {
                    if (!(e.bodyFlags[oj] & kOcculting) || oj == e.sunIndex) continue;
                    const double rB[3] = {pos[0] - r.body(oj, 0), pos[1] - r.body(oj, 1), pos[2] - r.body(oj, 2)};
                    occ *= shadowFactor(dp, rB, e.bodyRadius[bi], e.bodyRadius[oj]);
                }
            }
            const double f = occ * ((e.au * e.au * 4.56e-3 * ams) * (ird * ird * ird));
            ax += f * dp[0];
            ay += f * dp[1];
            az += f * dp[2];
        }
        if ((fl & kAtmosphere) && !isEarth && e.nExp > 0 && e.poleSlot[bi] >= 0) {
            // exponential drag in another body's atmosphere (PrivateAccelerations.h:143-204):
            // geodetic height about its polar axis, the air moving with its
            // rotation and its velocity relative to the Earth
            const int k = e.poleSlot[bi];
            const double d[3] = {pos[0] - rb[0], pos[1] - rb[1], pos[2] - rb[2]};
            const double pole[3] = {r.pole(k, 0), r.pole(k, 1), r.pole(k, 2)};
            const double h = geodeticHeight(d, pole, e.bodyRadius[bi], e.atmFlattening);
            int band = 0;
            for (int sgi = 1; sgi < e.nExp; ++sgi) band += e.expSeg[sgi][1] <= h ? 1 : 0;
            if (h <= e.expSeg[band][3]) {
                const double rho = e.expSeg[band][0] * exp(-(h - e.expSeg[band][1]) / e.expSeg[band][2]);
                const double w[3] = {r.poleW(k, 0), r.poleW(k, 1), r.poleW(k, 2)};
                const double vr0 = vel[0] - r.poleV(k, 0) - (w[1] * d[2] - w[2] * d[1]);
                const double vr1 = vel[1] - r.poleV(k, 1) - (w[2] * d[0] - w[0] * d[2]);
                const double vr2 = vel[2] - r.poleV(k, 2) - (w[0] * d[1] - w[1] * d[0]);
                const double f = -0.5 * rho * bc * sqrt(vr0 * vr0 + vr1 * vr1 + vr2 * vr2);
                ax += f * vr0;
                ay += f * vr1;
                az += f * vr2;
            }
        }
        if ((fl & kAtmosphere) && isEarth && !e.hasNrl && e.nExp > 0) {
            // piecewise exponential drag (PrivateAccelerations.h:137-206,
            // PiecewiseExponentialAtmosphere.h:40-90): band = bands above the
            // first whose base h0 <= h; no drag above the band's cut-off
            const double pole[3] = {r.R(6), r.R(7), r.R(8)};  // body z axis in inertial axes
            const double h = geodeticHeight(pos, pole, e.bodyRadius[bi], e.flattening);
            int band = 0;
            for (int sgi = 1; sgi < e.nExp; ++sgi) band += e.expSeg[sgi][1] <= h ? 1 : 0;
            if (h <= e.expSeg[band][3]) {
                const double rho = e.expSeg[band][0] * exp(-(h - e.expSeg[band][1]) / e.expSeg[band][2]);
                const double w[3] = {r.W(0), r.W(1), r.W(2)};
                const double vr0 = vel[0] - (w[1] * pos[2] - w[2] * pos[1]);
                const double vr1 = vel[1] - (w[2] * pos[0] - w[0] * pos[2]);
                const double vr2 = vel[2] - (w[0] * pos[1] - w[1] * pos[0]);
                const double f = -0.5 * rho * bc * sqrt(vr0 * vr0 + vr1 * vr1 + vr2 * vr2);
                ax += f * vr0;
                ay += f * vr1;
                az += f * vr2;
            }
        }
        if (NRL && (fl & kAtmosphere) && isEarth && e.hasNrl) {
            double rho;
            if constexpr (DUO) {
                duoSync(duo.barrier + 1);
                rho = duo.mail[(threadIdx.x & 31) / L].rho;
            } else {
                rho = nrlDensity<L>(e, r.nrlDeferred(), fb);
            }
            const double w[3] = {r.W(0), r.W(1), r.W(2)};
            const double vr0 = vel[0] - (w[1] * pos[2] - w[2] * pos[1]);
            const double vr1 = vel[1] - (w[2] * pos[0] - w[0] * pos[2]);
            const double vr2 = vel[2] - (w[0] * pos[1] - w[1] * pos[0]);
            const double f = -0.5 * rho * bc * sqrt(vr0 * vr0 + vr1 * vr1 + vr2 * vr2);
            ax += f * vr0;
            ay += f * vr1;
            az += f * vr2;
        }
    }
    if (e.tidesAlone) {
        double t[3] = {0.0, 0.0, 0.0};
        tideAloneAccel(r, pos, t);
        ax += t[0];
        ay += t[1];
        az += t[2];
    }
    if (e.relativity) {
        const double mu = tidefield::kMuEarth, c = tidefield::kLight;
        const double r0 = 1000.0 * pos[0], r1 = 1000.0 * pos[1], r2 = 1000.0 * pos[2];
        const double v0 = 1000.0 * vel[0], v1 = 1000.0 * vel[1], v2 = 1000.0 * vel[2];
        const double irr = rsqrt(r0 * r0 + r1 * r1 + r2 * r2);
        const double v2n = v0 * v0 + v1 * v1 + v2 * v2;
        const double rv = r0 * v0 + r1 * v1 + r2 * v2;
        const double f = mu * (irr * irr * irr) / (c * c);
        const double g = 4.0 * mu * irr - v2n;
        ax += 1.0e-3 * (f * (g * r0 + 4.0 * rv * v0));
        ay += 1.0e-3 * (f * (g * r1 + 4.0 * rv * v1));
        az += 1.0e-3 * (f * (g * r2 + 4.0 * rv * v2));
    }
    acc[0] = ax;
    acc[1] = ay;
    acc[2] = az;
}

// ---- TMA bulk staging of the coefficient tile --------------------------------------------------
// Stages the tile with bulk copies (32 KB chunks) on one mbarrier and waits
// for them with a bounded poll.  Returns whether the whole CTA saw the copies
// land; on a time-out the CTA reads the tile from global memory instead (the
// copies, should any still be in flight, only write the tile's region of
// shared memory, which the CTA then leaves alone).  `issue` = false arms the
// barrier without any copy (a test of the time-out path: nothing is in
// flight when the wait gives up).
static __device__ __forceinline__ bool stageTile(void* dst, const void* src, int bytes, bool issue, long polls) {
    __shared__ __align__(8) uint64_t bar;
    const uint32_t barAddr = (uint32_t)__cvta_generic_to_shared(&bar);
    const uint32_t dstAddr = (uint32_t)__cvta_generic_to_shared(dst);
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(barAddr));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(barAddr), "r"(bytes) : "memory");
        const int chunk = 32768;
        for (int off = 0; issue && off < bytes; off += chunk) {
            const int sz = (bytes - off) < chunk ? (bytes - off) : chunk;
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                    dstAddr + off),
                "l"((const char*)src + off), "r"(sz), "r"(barAddr)
                : "memory");
        }
    }
    __syncthreads();
    // bounded wait on phase 0
    uint32_t done = 0;
    for (long it = 0; it < polls && !done; ++it) {
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
            : "=r"(done)
            : "r"(barAddr), "r"(0)
            : "memory");
    }
    return __syncthreads_and((int)done) != 0;
}

// ---- the persistent step kernel ----------------------------------------------------------------
// Stage record of a per-object-time batch: 4-point Lagrange weights in the
// batch's record grid (rotation, angular velocity, body positions, tide
// deltas; a 30 s spacing keeps the interpolation error of the rotation below
// 1e-12 relative), read field by field by the force model; the NRLMSISE-00
// time inputs are evaluated exactly at the stage epoch by the drag model
// when it needs them.
static __device__ __forceinline__ RecordInterp recordFromGrid(const StepParams& p, double et) {
    // stencil k0 - 1 .. k0 + 2 around the absolute grid index k0 = floor(et / H);
    // q depends on et alone, so the weights are the same in every batch
    const double u = et / p.gridH;
    const double kf = floor(u);
    int64_t i0 = (int64_t)kf - 1 - p.gridBase;
    i0 = i0 < 0 ? 0 : (i0 > p.gridN - 4 ? p.gridN - 4 : i0);
    const double q = u - kf + 1.0;
    double w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        double num = 1.0, den = 1.0;
#pragma unroll
        for (int m = 0; m < 4; ++m)
            if (m != j) {
                num *= q - (double)m;
                den *= (double)(j - m);
            }
        w[j] = num / den;
    }
    return RecordInterp{p.gridPairs + i0 * kInterpFields, w[0], w[1], w[2], w[3], et};
}

// MAXT: the thread bound the kernel is compiled for, which sets its register
// budget (the register file is split over the SM's four sub-partitions, so
// 320 or 384 threads leave 168 registers a thread and 256 threads leave 255).
// STREAM: the tile streamed through rings (TileStream).  DUO: warps in pairs,
// the drag model on the second (duoPartner).  NRL: with NRLMSISE-00; that
// model is most of the kernel's code and holds most of its spilled state, so
// configurations without it run kernels without it (333 objects on J2-J6 x 60
// steps 1.50 -> 1.41 ms, the field alone on 5,000 x 10 2.62 -> 2.49).
template <int L, typename T, bool SHARED_GRID, bool PAIR, int MAXT, bool STREAM, bool NRL, bool DUO>
__global__ void __launch_bounds__(MAXT, 1) propagateKernel(const __grid_constant__ StepParams p) {
    constexpr TileRead MODE = STREAM                ? TileRead::kStream
                              : MAXT <= kDeepThreads ? TileRead::kShared
                                                     : TileRead::kGeneric;
    constexpr int NA = Axes<L>::N;
    TileRef tile{p.tile, p.nblocks, 0};
    int kOffset = 0;
    if (!SHARED_GRID && !p.gridPairs) {  // per-object time needs the batch's record grid
        if (threadIdx.x == 0) atomicExch(p.errorFlag, 3);
        return;
    }
    if (!STREAM && p.useSmemTile) {
        const bool test = p.tileWaitTest != 0;
        if (stageTile(g_smem, p.tile, p.stagedBytes, !test, test ? 4096L : (1L << 24)))
            tile.staged = p.stagedBytes / 16;
        else if (threadIdx.x == 0 && p.tileFallbacks)
            atomicAdd(p.tileFallbacks, 1);  // this CTA reads the tile from global memory
        kOffset = p.stagedBytes;
    }
    // main warps of the CTA and this warp's place among them
    const int warps = (int)(blockDim.x / 32) / (DUO ? 2 : 1), warp = (int)(threadIdx.x / 32) / (DUO ? 2 : 1);
    Duo duo{nullptr, nullptr, 0};
    if constexpr (DUO) {
        __shared__ DuoMail s_mail[kDuoPairs][32 / L];
        __shared__ int s_quit[kDuoPairs];
        duo = Duo{s_mail[warp], &s_quit[warp], 1 + 2 * warp};
        if (threadIdx.x % 64 == 0) s_quit[warp] = 0;
        __syncthreads();
        if ((threadIdx.x / 32) & 1) {
            duoPartner<L>(p.env, duo);
            return;
        }
    }
    TileStream<(PAIR ? 2 : 1) * L> stream;
    if constexpr (STREAM) {
        stream.begin(warp * kRingBytes, p.tile, p.tileBytes);
        kOffset = warps * kRingBytes;
    }
    const StageStore kst{(double*)(g_smem + kOffset) + (warp * 32 + (int)(threadIdx.x & 31)) / L, warps * 32 / L};
    const int lane = (int)(threadIdx.x & 31);
    const int j = lane % L;
    const int g = lane / L;
    constexpr int groups = 32 / L;
    const int groupBase = lane - j;
    // Work items are groups of 32/L consecutive objects (in the processing
    // order, i.e. by altitude).  The first wave is assigned statically with
    // consecutive items on different CTAs, so the costly low-altitude groups
    // spread over all SMs instead of landing on the CTAs that start first;
    // later items come from the atomic queue.
    const int64_t nItems = (p.n + groups - 1) / groups;
    const int64_t firstWave = (int64_t)gridDim.x * warps;
    auto nextItem = [&]() {
        int64_t next = 0;
        if (lane == 0) next = firstWave + (int64_t)atomicAdd(p.workCounter, 1);
        return __shfl_sync(0xffffffffu, next, 0);
    };
    for (int64_t item = (int64_t)warp * gridDim.x + blockIdx.x; item < nItems; item = nextItem()) {
        const int64_t base = item * groups;
        const int64_t slot = base + g;
        const bool valid = slot < p.n;
        const int64_t sidx = valid ? slot : p.n - 1;
        const int64_t oi = p.order ? p.order[sidx] : sidx;
        const int64_t stride = p.stride ? p.stride : p.n;
        double y[NA], v[NA];
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            const int axis = Axes<L>::axis(j, i);
            y[i] = p.state[(int64_t)axis * stride + oi];
            v[i] = p.state[(int64_t)(axis + 3) * stride + oi];
        }
        const double bc = p.bc[oi], ams = p.ams[oi];
        double cur = 0.0, dtv = 0.0, endv = 0.0, stepv = 0.0;
        bool done = false;
        if (!SHARED_GRID) {
            cur = p.cur[oi];
            dtv = p.dt[oi];
            endv = p.end[oi];
            stepv = p.step[oi];
            done = !valid || !(dtv > 0.0);  // a resident batch keeps objects that have reached their end
        }
        const int64_t nsteps = SHARED_GRID ? (int64_t)p.nsteps : p.maxSteps;
        for (int64_t kstep = 0; kstep < nsteps; ++kstep) {
            if (!SHARED_GRID) {
                if (!__any_sync(0xffffffffu, !done)) break;
            }
            const double t0 = SHARED_GRID ? p.stepT0[kstep] : cur;
            const double dt = SHARED_GRID ? p.stepDt[kstep] : dtv;
            double acc[3];
            // one copy of the force model: the stage loop is not unrolled
#pragma unroll 1
            for (int s = 0; s < 13; ++s) {
                double ys[NA], vs[NA];
                switch (s) {
                    case 0:
#pragma unroll
                        for (int i = 0; i < NA; ++i) {
                            ys[i] = y[i];
                            vs[i] = v[i];
                        }
                        break;
                    case 1: stageState<L, 1>(y, v, kst, j, dt, ys, vs); break;
                    case 2: stageState<L, 2>(y, v, kst, j, dt, ys, vs); break;
                    case 3: stageState<L, 3>(y, v, kst, j, dt, ys, vs); break;
                    case 4: stageState<L, 4>(y, v, kst, j, dt, ys, vs); break;
                    case 5: stageState<L, 5>(y, v, kst, j, dt, ys, vs); break;
                    case 6: stageState<L, 6>(y, v, kst, j, dt, ys, vs); break;
                    case 7: stageState<L, 7>(y, v, kst, j, dt, ys, vs); break;
                    case 8: stageState<L, 8>(y, v, kst, j, dt, ys, vs); break;
                    case 9: stageState<L, 9>(y, v, kst, j, dt, ys, vs); break;
                    case 10: continue;  // enters neither a stage nor the update
                    case 11: stageState<L, 11>(y, v, kst, j, dt, ys, vs); break;
                    default: stageState<L, 12>(y, v, kst, j, dt, ys, vs); break;
                }
                double st[6];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const double py = ys[Axes<L>::place(a)], pv = vs[Axes<L>::place(a)];
                    st[a] = L == 1 ? py : __shfl_sync(0xffffffffu, py, groupBase + Axes<L>::lane(a));
                    st[a + 3] = L == 1 ? pv : __shfl_sync(0xffffffffu, pv, groupBase + Axes<L>::lane(a));
                }
                if (SHARED_GRID) {
                    const RecordRef rec{p.records + kstep * 13 + s};
                    // the next record's lines on their way to L1 (each stage
                    // reads its record at half a dozen points of the force
                    // model, a trip to L2 at each otherwise: 1,024 objects x
                    // 10 steps on the point mass 0.148 -> 0.129 ms, 333 on
                    // J2-J6 x 60 1.69 -> 1.52); the last stage of all reads
                    // its own again
                    {
                        const bool final = s == 12 && kstep + 1 == nsteps;
                        const char* nextRec = (const char*)(rec.r + (final ? 0 : s == 9 ? 2 : 1));
                        constexpr int kLines = (int)(sizeof(EpochRecord) + 127) / 128;
                        if (lane < kLines) {
                            unsigned touch;
                            asm volatile("ld.global.ca.u32 %0, [%1];"
                                         : "=r"(touch)
                                         : "l"(nextRec + (lane * 128 < (int)sizeof(EpochRecord) - 4 ? lane * 128 : 0)));
                        }
                    }
                    accelerations<L, T, PAIR, MODE, NRL, DUO>(p, tile, stream, duo, rec, st, st + 3, bc, ams, acc);
                } else {
                    const double ts = s == 0 ? t0 : t0 + dt * rkC(s - 1);
                    const RecordInterp rec = recordFromGrid(p, ts);
                    accelerations<L, T, PAIR, MODE, NRL, DUO>(p, tile, stream, duo, rec, st, st + 3, bc, ams, acc);
                }
                if (s < 12) {
#pragma unroll
                    for (int i = 0; i < NA; ++i) {
                        const int axis = Axes<L>::axis(j, i);
                        if (Axes<L>::writes(j, i))
                            kst.at(rkSlot(s), axis) = axis == 0 ? acc[0] : axis == 1 ? acc[1] : acc[2];
                    }
                    if (L > 1) __syncwarp();
                }
            }
            finalUpdate<L>(y, v, kst, j, dt, acc, SHARED_GRID || !done);
            if (L > 1) __syncwarp();
            if (SHARED_GRID && p.traj && (kstep + 1) % p.trajEvery == 0 && valid
                && (kstep + 1) / p.trajEvery <= p.trajRecords) {
                double* rec = p.traj + (int64_t)((kstep + 1) / p.trajEvery - 1) * 6 * p.n;
#pragma unroll
                for (int i = 0; i < NA; ++i) {
                    const int axis = Axes<L>::axis(j, i);
                    if (Axes<L>::writes(j, i)) {
                        rec[(int64_t)axis * p.n + oi] = y[i];
                        rec[(int64_t)(axis + 3) * p.n + oi] = v[i];
                    }
                }
            }
            if (!SHARED_GRID && !done) {
                // FixedStep.h:30-37
                cur += dtv;
                const double rem = endv - cur;
                done = rem <= 0;
                dtv = done ? 0.0 : fmin(stepv, rem);
            }
        }
        if (valid) {
#pragma unroll
            for (int i = 0; i < NA; ++i) {
                const int axis = Axes<L>::axis(j, i);
                if (Axes<L>::writes(j, i)) {
                    p.state[(int64_t)axis * stride + oi] = y[i];
                    p.state[(int64_t)(axis + 3) * stride + oi] = v[i];
                }
            }
            if (!SHARED_GRID && j == 0) {
                p.cur[oi] = cur;
                p.dt[oi] = dtv;
                p.unfinished[oi] = done ? 0 : 1;
            }
        }
    }
    if constexpr (DUO) {
        if ((threadIdx.x & 31) == 0) *duo.quit = 1;
        duoArrive(duo.barrier);
    }
    if constexpr (STREAM) stream.end();
}

}  // namespace phop

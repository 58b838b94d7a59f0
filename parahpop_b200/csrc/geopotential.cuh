// Geopotential of the step kernel: the field's acceleration from the
// coefficient tile (geopotential.hpp) and the Earth's tide deltas.
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

#include "geopotential.hpp"
#include "propagate.cuh"

namespace phop {

// Two FP32 values in one 64-bit register pair, operated on by the packed
// f32x2 instructions of sm_100.
struct F2 {
    unsigned long long v;
};
static __device__ __forceinline__ F2 f2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}

// K objects' values of one lane, operated on together.  The roundings are
// explicit (__fma_rn, __dmul_rn and so on): an object's result must not
// depend on which of the K places it takes, that is, on which other objects
// share its warp, so nothing is left to the compiler's contraction of each
// place's copy of the code.
template <typename T, int K> struct Lanes;
template <int K> struct Lanes<double, K> {
    double v[K];
    static __device__ __forceinline__ Lanes all(double a) {
        Lanes r;
#pragma unroll
        for (int k = 0; k < K; ++k) r.v[k] = a;
        return r;
    }
    __device__ __forceinline__ void set(int k, double a) { v[k] = a; }
    __device__ __forceinline__ double get(int k) const { return v[k]; }
};
template <int K>
static __device__ __forceinline__ Lanes<double, K> vfma(double a, const Lanes<double, K>& b, const Lanes<double, K>& c) {
    Lanes<double, K> r;
#pragma unroll
    for (int k = 0; k < K; ++k) r.v[k] = __fma_rn(a, b.v[k], c.v[k]);
    return r;
}
// w = a u; returns w q + t q1 with t = -alpha^2
template <int K>
static __device__ __forceinline__ Lanes<double, K> vstep(double a, const Lanes<double, K>& u, const Lanes<double, K>& q,
                                                         const Lanes<double, K>& t, const Lanes<double, K>& q1) {
    Lanes<double, K> r;
#pragma unroll
    for (int k = 0; k < K; ++k)
        r.v[k] = __fma_rn(__dmul_rn(a, u.v[k]), q.v[k], __dmul_rn(t.v[k], q1.v[k]));
    return r;
}
template <> struct Lanes<float, 1> {
    float v;
    static __device__ __forceinline__ Lanes all(float a) { return Lanes{a}; }
    __device__ __forceinline__ void set(int, double a) { v = (float)a; }
    __device__ __forceinline__ double get(int) const { return (double)v; }
};
static __device__ __forceinline__ Lanes<float, 1> vfma(float a, Lanes<float, 1> b, Lanes<float, 1> c) {
    return Lanes<float, 1>{__fmaf_rn(a, b.v, c.v)};
}
static __device__ __forceinline__ Lanes<float, 1> vstep(float a, Lanes<float, 1> u, Lanes<float, 1> q, Lanes<float, 1> t,
                                                        Lanes<float, 1> q1) {
    return Lanes<float, 1>{__fmaf_rn(__fmul_rn(a, u.v), q.v, __fmul_rn(t.v, q1.v))};
}
template <> struct Lanes<float, 2> {
    F2 v;
    static __device__ __forceinline__ Lanes all(float a) { return Lanes{f2(a, a)}; }
    __device__ __forceinline__ void set(int k, double a) {
        float lo, hi;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v.v));
        v = k == 0 ? f2((float)a, hi) : f2(lo, (float)a);
    }
    __device__ __forceinline__ double get(int k) const {
        float lo, hi;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v.v));
        return (double)(k == 0 ? lo : hi);
    }
};
static __device__ __forceinline__ F2 f2fma(F2 a, F2 b, F2 c) {
    F2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return d;
}
static __device__ __forceinline__ F2 f2mul(F2 a, F2 b) {
    F2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
    return d;
}
static __device__ __forceinline__ Lanes<float, 2> vfma(float a, Lanes<float, 2> b, Lanes<float, 2> c) {
    return Lanes<float, 2>{f2fma(f2(a, a), b.v, c.v)};
}
static __device__ __forceinline__ Lanes<float, 2> vstep(float a, Lanes<float, 2> u, Lanes<float, 2> q, Lanes<float, 2> t,
                                                        Lanes<float, 2> q1) {
    return Lanes<float, 2>{f2fma(f2mul(f2(a, a), u.v), q.v, f2mul(t.v, q1.v))};
}

// One row: the six sums take q, then q advances (q1 holds the value before).
template <typename T, int K>
static __device__ __forceinline__ void fieldRow(T a, T xc, T xs, T yc, T ys, T zc, T zs, const Lanes<T, K>& u,
                                                const Lanes<T, K>& t, Lanes<T, K>& q, Lanes<T, K>& q1,
                                                Lanes<T, K> (&S)[6]) {
    S[0] = vfma(xc, q, S[0]);
    S[1] = vfma(xs, q, S[1]);
    S[2] = vfma(yc, q, S[2]);
    S[3] = vfma(ys, q, S[3]);
    S[4] = vfma(zc, q, S[4]);
    S[5] = vfma(zs, q, S[5]);
    const Lanes<T, K> n = vstep(a, u, q, t, q1);
    q1 = q;
    q = n;
}

// The tile: staged at the start of the CTA's dynamic shared memory, streamed
// through the warp's ring (kernels that read shared memory by their own
// loads), or read from global memory.
extern __shared__ __align__(128) unsigned char g_smem[];
struct TileRef {
    const void* global;
    int nblocks;
    int staged;  // 16-byte chunks staged: whole blocks from the tile's start
};

// The stream of a tile too large for shared memory: the warp copies it, stage
// by stage (2 KiB, four 16-byte cp.async a lane), into a ring of eight stages
// in shared memory, always five to six stages ahead of its row loop, and
// starts over at the tile's end for the next evaluation.  A row (W chunks)
// may be read once `ready` has passed it.  Stage k is acquired while the
// reading row is in stage k - 1 at the earliest, so the slot of stage k - 2
// is free then and takes the next copy.  The ring's first rows are repeated
// past its end, so that a row pair is read at fixed offsets from its first
// row.  Every lane of the warp makes every call.  The loads of a warp then
// come from shared memory with hundreds of cycles of lead, instead of missing
// L1 one row pair at a time: 10^5 LEO objects x 4 steps at degree 120 in
// split precision 37.9 -> 26.7 ms, 20,011 in FP64 13.6 -> 11.1 (four
// lanes; one lane 20.4 -> 13.1).
template <int W>
struct TileStream {
    static constexpr unsigned kRows = kStageChunks / W;  // rows of a stage
    static constexpr unsigned kMask = kRingStages * kRows - 1;
    int base = 0;  // byte offset of the ring in g_smem
    const uint4* src = nullptr;
    int stages = 0, next = 0;
    unsigned issued = 0, pos = 0, ready = 0;

    __device__ __forceinline__ void issue() {
        static_assert(W > 8 || 2 * kChunks64 <= kRows, "a stage holds two row pairs");
        const int lane = (int)(threadIdx.x & 31), slot = (int)(issued & (kRingStages - 1));
        const uint4* from = src + (size_t)next * kStageChunks + lane;
        const uint32_t to = (uint32_t)__cvta_generic_to_shared(g_smem) + base + (slot * kStageChunks + lane) * 16;
#pragma unroll
        for (int i = 0; i < kStageChunks / 32; ++i)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + i * 512), "l"(from + i * 32) : "memory");
        if (slot == 0) {
#pragma unroll
            for (int i = 0; i < (kRingMirror * W + 31) / 32; ++i)
                if (lane + i * 32 < kRingMirror * W)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + kRingStages * kStageChunks * 16
                                                                                   + i * 512),
                                 "l"(from + i * 32)
                                 : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        next = next + 1 == stages ? 0 : next + 1;
        ++issued;
    }
    __device__ __forceinline__ void begin(int smemOffset, const void* tile, int bytes) {
        base = smemOffset;
        src = (const uint4*)tile;
        stages = bytes / (kStageChunks * 16);
        for (int k = 0; k < kRingStages - 2; ++k) issue();
    }
    // rows pos .. pos + rows - 1 readable (rows <= kRows)
    __device__ __forceinline__ void need(unsigned rows) {
        if ((int)(pos + rows - ready) > 0) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kRingStages - 3) : "memory");
            __syncwarp();
            issue();
            ready += kRows;
        }
    }
    // the lane's chunk of the row `ahead` rows on
    template <typename Chunk> __device__ __forceinline__ const Chunk* row(unsigned ahead, int pj) const {
        return (const Chunk*)(g_smem + base) + ((pos + ahead) & kMask) * W + pj;
    }
    // the tile's padding at the end of an evaluation
    __device__ __forceinline__ void rewind() { pos = ready; }
    __device__ __forceinline__ void end() {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
};

// The chunks of one row pair of a lane, W lanes interleaved.
template <typename T> struct PairRows;
template <> struct PairRows<double> {
    static constexpr int kChunks = kChunks64;
    double2 c[kChunks64];
    template <int W> __device__ __forceinline__ void load(const double2* __restrict__ tp) {
#pragma unroll
        for (int i = 0; i < kChunks64; ++i) c[i] = tp[i * W];
    }
    template <int K>
    __device__ __forceinline__ void add(const Lanes<double, K>& u, const Lanes<double, K>& t, Lanes<double, K>& q,
                                        Lanes<double, K>& q1, Lanes<double, K> (&S)[6]) const {
        fieldRow<double, K>(c[0].x, c[1].x, c[1].y, c[2].x, c[2].y, c[3].x, c[3].y, u, t, q, q1, S);
        fieldRow<double, K>(c[0].y, c[4].x, c[4].y, c[5].x, c[5].y, c[6].x, c[6].y, u, t, q, q1, S);
    }
};
template <> struct PairRows<float> {
    static constexpr int kChunks = kChunks32;
    float4 a, b, c;
    float2 d;
    template <int W> __device__ __forceinline__ void load(const float4* __restrict__ tp) {
        a = tp[0];
        b = tp[W];
        c = tp[2 * W];
        d = *(const float2*)(tp + 3 * W);
    }
    template <int K>
    __device__ __forceinline__ void add(const Lanes<float, K>& u, const Lanes<float, K>& t, Lanes<float, K>& q,
                                        Lanes<float, K>& q1, Lanes<float, K> (&S)[6]) const {
        fieldRow<float, K>(a.x, a.z, a.w, b.x, b.y, b.z, b.w, u, t, q, q1, S);
        fieldRow<float, K>(a.y, c.x, c.y, c.z, c.w, d.x, d.y, u, t, q, q1, S);
    }
};
// `pairs` row pairs of a column from its first 16-byte chunk.  kShared: a staged tile is
// read by shared-memory loads, in a loop of its own, two row pairs an
// iteration (four measured better in FP32 by itself, 82.7 against 85.7
// thousand cycles an evaluation at degree 70, but worse in the whole kernel,
// whose instructions it crowds: 10^6 uneven objects 109 against 103 ms).  Such a load whose lanes differ in at most two addresses (W <=
// 2) takes 2 cycles of an SM per 16 bytes of a warp, a generic load 4, and
// the column loop of one lane per object was bound by the latter (82 % of the
// load path's peak, FP64 pipe 52 %): 200,000 uneven objects x 8 steps FP64
// 66.3 -> 60.5 ms, 10^6 x 4 split 110 -> 100; at four lanes the shorter
// latency shows, 10^4 LEO x 20 FP64 14.9 -> 13.7.  The kernels of 168
// registers keep one generic loop: with two they spill inside them (two
// lanes, pairs, 10^4 LEO: 21.0 against 27.0 ms).
// `room`: the pairs the block holds per lane (the stream passes them all);
// ALL: pairs == room.
enum class TileRead { kGeneric, kShared, kStream };  // see fieldRows; the kernel's instantiation
template <typename T, int K, int W, TileRead MODE, bool ALL>
static __device__ __forceinline__ void fieldRows(const TileRef& tile, TileStream<W>& stream, int pj, int chunk, int pairs,
                                                 int room, const Lanes<T, K>& u, const Lanes<T, K>& t, Lanes<T, K>& q,
                                                 Lanes<T, K>& q1, Lanes<T, K> (&S)[6]) {
    using Chunk = typename std::conditional<sizeof(T) == 8, double2, float4>::type;
    constexpr int kChunks = PairRows<T>::kChunks, kStep = kChunks * W;
    // the shapes that may hold a part of the tile (hasPart) ask block by block;
    // asked in the others too, it cost the field alone of 5,000 objects 3.5 %
    constexpr bool kPart = MODE == TileRead::kGeneric || (K == 1 && W >= 8);
    const bool staged = kPart ? chunk < tile.staged : tile.staged != 0;
    if (MODE == TileRead::kShared && staged) {
        const Chunk* tp = (const Chunk*)g_smem + chunk + pj;
#pragma unroll 2
        for (int i = 0; i < pairs; ++i, tp += kStep) {
            PairRows<T> r;
            r.template load<W>(tp);
            r.template add<K>(u, t, q, q1, S);
        }
        return;
    }
    if constexpr (MODE == TileRead::kStream) {
        int i = 0;
        for (; i + 1 < room; i += 2) {
            stream.need(2 * kChunks);
            PairRows<T> r0, r1;
            r0.template load<W>(stream.template row<Chunk>(0, pj));
            r1.template load<W>(stream.template row<Chunk>(kChunks, pj));
            stream.pos += 2 * kChunks;
            if (ALL || i < pairs) r0.template add<K>(u, t, q, q1, S);
            if (ALL || i + 1 < pairs) r1.template add<K>(u, t, q, q1, S);
        }
        if (i < room) {
            stream.need(kChunks);
            PairRows<T> r;
            r.template load<W>(stream.template row<Chunk>(0, pj));
            stream.pos += kChunks;
            if (ALL || i < pairs) r.template add<K>(u, t, q, q1, S);
        }
        return;
    }
    const Chunk* __restrict__ tp =
        (const Chunk*)(MODE == TileRead::kGeneric && staged ? (const void*)g_smem : tile.global) + chunk + pj;
    for (int i = 0; i < pairs; ++i, tp += kStep) {
        PairRows<T> r;
        r.template load<W>(tp);
        r.template add<K>(u, t, q, q1, S);
    }
}

// Per-object quantities of the column sums.
struct FieldGeo {
    double u, t;          // alpha sin phi, -alpha^2
    double cL, sL, mag;   // cos, sin of M lambda; (alpha cos phi)^M
    double cW, sW, magW;  // the same for W orders
    double acc[3];
};

// the calling lane's first column is M = first; columns then advance by W
template <int W>
static __device__ __forceinline__ void fieldGeo(double x, double y, double z, double R, int first, FieldGeo& g) {
    const double rho2 = __fma_rn(y, y, __dmul_rn(x, x));
    const double rn = __dsqrt_rn(__fma_rn(z, z, rho2)), rho = __dsqrt_rn(rho2);
    const double inv = __drcp_rn(rn), alpha = __dmul_rn(R, inv);
    g.u = __dmul_rn(alpha, __dmul_rn(z, inv));
    g.t = -__dmul_rn(alpha, alpha);
    g.cW = 1.0;
    g.sW = 0.0;
    if (rho > 1e-14) {
        const double ir = __drcp_rn(rho);
        g.cW = __dmul_rn(x, ir);
        g.sW = __dmul_rn(y, ir);
    }
    g.magW = __dmul_rn(alpha, __dmul_rn(rho, inv));
    g.cL = 1.0;
    g.sL = 0.0;
    g.mag = 1.0;
    // powers by squaring: order `first` for the lane, order W for the step
#pragma unroll
    for (int bit = 1; bit < W; bit <<= 1) {
        if (first & bit) {
            const double c = __fma_rn(g.cW, g.cL, -__dmul_rn(g.sW, g.sL));
            g.sL = __fma_rn(g.cW, g.sL, __dmul_rn(g.sW, g.cL));
            g.cL = c;
            g.mag = __dmul_rn(g.mag, g.magW);
        }
        const double c = __fma_rn(g.cW, g.cW, -__dmul_rn(g.sW, g.sW));
        g.sW = __dmul_rn(2.0, __dmul_rn(g.sW, g.cW));
        g.cW = c;
        g.magW = __dmul_rn(g.magW, g.magW);
    }
    g.acc[0] = g.acc[1] = g.acc[2] = 0.0;
}

// Earth's tide deltas (n = 2..6, fully normalised, field units): the part of
// lane j of the object's L lanes (orders m = j, j + L, ... <= 6), in the
// units of the field's column sums.  Pines' form (AIAA J. 11(11),
// 1973): with A_nm = P_nm / cos^m phi and (r_m + i i_m) = ((x + i y)/r)^m,
//   a1 = sum m A (C r_{m-1} + S i_{m-1}),  a2 = sum m A (S r_{m-1} - C i_{m-1}),
//   a3 = sum k A_{n,m+1} (C r_m + S i_m),  a4 = -sum ((n+m+1) A + u k A_{n,m+1}) (C r_m + S i_m),
//   acc = (a1 + s a4, a2 + t a4, a3 + u a4), each term weighted by alpha^n.
// No pole case.  A column's deltas are read before they are used, so that
// their loads overlap (a rolled loop of dependent reads cost more than the
// sums).
struct TideStep {
    double a, b, e, k;  // A_n = a u A_{n-1} - b A_{n-2} + e; k: A_{n,m+1} against the latitude derivative of A_nm
};
// orders 0..7, degrees 2..6 (order 7 has none: the latitude neighbour of order 6)
static __device__ const TideStep g_tideStep[8][5] = {
    {{1.9364916731037085, 1.118033988749895, 0.0, 1.7320508075688772},
     {1.9720265943665387, 1.0183501544346312, 0.0, 2.449489742783178},
     {1.984313483298443, 1.0062305898749053, 0.0, 3.1622776601683795},
     {1.98997487421324, 1.002853072844814, 0.0, 3.872983346207417},
     {1.9930434571835662, 1.0015420209622192, 0.0, 4.58257569495584}},
    {{2.23606797749979, 0.0, 0.0, 2.0},
     {2.091650066335189, 0.9354143466934853, 0.0, 3.1622776601683795},
     {2.04939015319192, 0.9797958971132712, 0.0, 4.242640687119285},
     {2.03100960115899, 0.9910312089651149, 0.0, 5.291502622129181},
     {2.0213149892370277, 0.9952267030562386, 0.0, 6.324555320336759}},
    {{0.0, 0.0, 1.9364916731037085, 0.0},
     {2.6457513110645907, 0.0, 0.0, 2.449489742783178},
     {2.29128784747792, 0.8660254037844386, 0.0, 3.7416573867739413},
     {2.1712405933672376, 0.9476070829586857, 0.0, 4.898979485566356},
     {2.1139418156609704, 0.9736101204623269, 0.0, 6.0}},
    {{0.0, 0.0, 0.0, 0.0},
     {0.0, 0.0, 2.091650066335189, 0.0},
     {3.0, 0.0, 0.0, 2.8284271247461903},
     {2.48746859276655, 0.82915619758885, 0.0, 4.242640687119285},
     {2.3013683530231086, 0.9251848886516145, 0.0, 5.477225575051661}},
    {{0.0, 0.0, 0.0, 0.0},
     {0.0, 0.0, 0.0, 0.0},
     {0.0, 0.0, 2.218529918662356, 0.0},
     {3.3166247903554, 0.0, 0.0, 3.1622776601683795},
     {2.6739483914241875, 0.8062257748298549, 0.0, 4.69041575982343}},
    {{0.0, 0.0, 0.0, 0.0},
     {0.0, 0.0, 0.0, 0.0},
     {0.0, 0.0, 0.0, 0.0},
     {0.0, 0.0, 2.3268138086232857, 0.0},
     {3.605551275463989, 0.0, 0.0, 3.4641016151377544}},
    {{0.0, 0.0, 0.0, 0.0},
     {0.0, 0.0, 0.0, 0.0},
     {0.0, 0.0, 0.0, 0.0},
     {0.0, 0.0, 0.0, 0.0},
     {0.0, 0.0, 2.4218245962496954, 0.0}},
    {{0.0, 0.0, 0.0, 0.0},
     {0.0, 0.0, 0.0, 0.0},
     {0.0, 0.0, 0.0, 0.0},
     {0.0, 0.0, 0.0, 0.0},
     {0.0, 0.0, 0.0, 0.0}}};

template <int L, class Rec>
static __device__ __forceinline__ void tidePart(const Rec& rec, int j, double x, double y, double z, double R,
                                                double acc[3]) {
    const double inv = __drcp_rn(__dsqrt_rn(__fma_rn(z, z, __fma_rn(y, y, __dmul_rn(x, x)))));
    const double s = __dmul_rn(x, inv), t = __dmul_rn(y, inv), u = __dmul_rn(z, inv);
    const double alpha = __dmul_rn(R, inv);
    double a1 = 0.0, a2 = 0.0, a3 = 0.0, a4 = 0.0;
    // (r, i) of order m - 1 and m
    double rp = 0.0, ip = 0.0, r = 1.0, i = 0.0;
    auto turn = [&]() {
        rp = r;
        ip = i;
        r = __fma_rn(s, rp, -__dmul_rn(t, ip));
        i = __fma_rn(s, ip, __dmul_rn(t, rp));
    };
    for (int k = 0; k < j && k < 7; ++k) turn();
    constexpr double kA11 = 1.7320508075688772;  // sqrt(3)
#pragma unroll 1
    for (int m = j; m <= 6; m += L) {
        double c[5], d[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            const int n = q + 2;
            const bool on = n >= m;
            c[q] = on ? rec.dC(n * (n + 1) / 2 + m) : 0.0;
            d[q] = on && m > 0 ? rec.dS(n * (n + 1) / 2 + m) : 0.0;
        }
        // A_nm and A_{n,m+1}
        double p1 = m == 0 ? __dmul_rn(kA11, u) : m == 1 ? kA11 : 0.0, p0 = m == 0 ? 1.0 : 0.0;
        double h1 = m == 0 ? kA11 : 0.0, h0 = 0.0;
        double rho = alpha;
        double Fc = 0, Fs = 0, Gc = 0, Gs = 0, Hc = 0, Hs = 0;
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            const TideStep f = g_tideStep[m][q], g = g_tideStep[m + 1][q];
            const double p = __fma_rn(__dmul_rn(f.a, u), p1, __fma_rn(-f.b, p0, f.e));
            const double h = __fma_rn(__dmul_rn(g.a, u), h1, __fma_rn(-g.b, h0, g.e));
            p0 = p1;
            p1 = p;
            h0 = h1;
            h1 = h;
            rho = __dmul_rn(rho, alpha);
            const double A = __dmul_rn(rho, p), H = __dmul_rn(rho, __dmul_rn(f.k, h));
            const double G = __dmul_rn((double)(q + 3 + m), A);
            Fc = __fma_rn(c[q], A, Fc);
            Fs = __fma_rn(d[q], A, Fs);
            Gc = __fma_rn(c[q], G, Gc);
            Gs = __fma_rn(d[q], G, Gs);
            Hc = __fma_rn(c[q], H, Hc);
            Hs = __fma_rn(d[q], H, Hs);
        }
        const double dm = (double)m;
        a1 = __fma_rn(dm, __fma_rn(Fc, rp, __dmul_rn(Fs, ip)), a1);
        a2 = __fma_rn(dm, __fma_rn(Fs, rp, -__dmul_rn(Fc, ip)), a2);
        const double D3 = __fma_rn(Hc, r, __dmul_rn(Hs, i));
        a3 = __dadd_rn(a3, D3);
        a4 = __dsub_rn(a4, __fma_rn(u, D3, __fma_rn(Gc, r, __dmul_rn(Gs, i))));
        if (m + L <= 6) {
#pragma unroll 1
            for (int k = 0; k < L; ++k) turn();
        }
    }
    // to the units of the field's column sums (GM / R^2 alpha comes at the end)
    acc[0] = __dmul_rn(alpha, __fma_rn(s, a4, a1));
    acc[1] = __dmul_rn(alpha, __fma_rn(t, a4, a2));
    acc[2] = __dmul_rn(alpha, __fma_rn(u, a4, a3));
}

// Acceleration (body frame, km/s^2) of the calling lane's object at body-frame
// position (x, y, z), the same on every lane of its group of L lanes.  K
// groups of L lanes form a set of W = K L lanes: every lane takes the orders
// M = b W + (its place in the set) for all K objects of the set, so a loaded
// coefficient serves K objects.  Returns through `out`.
//
// Shared memory delivers 128 bytes a cycle to an SM's registers, whatever
// the lanes share (measured: 4.0 cycles per 16-byte load of a warp, 2.2 when
// at most two addresses differ), and the FP64 units take a warp's
// instruction in 2 cycles per quarter SM: a row's 56 bytes cost 14 cycles
// (7.7 at W <= 2) against 4.5 cycles of FP64 work per object, so one object a
// lane is bound by shared memory and two are near balance.  Step kernel, ms
// before (spherical components: 15 operations and 48 bytes a term) and now,
// each at its best shape: 10^4 LEO objects x 20 steps at degree 70 FP64 20.1
// -> 16.2, split 19.3 -> 13.9; 200,000 uneven objects x 8 steps FP64 121 ->
// 86.6; 10^6 x 4 split 239 -> 126; 10^5 LEO x 4 at degree 120 split 62 -> 37.
template <int L, int K, typename T, TileRead MODE, class Rec>
static __device__ __forceinline__ void fieldAccel(const StepParams& p, const TileRef& tile, TileStream<K * L>& stream,
                                                  const Rec& rec, double x, double y, double z, double out[3]) {
    constexpr int W = K * L;
    constexpr bool kSplit = sizeof(T) == 4;
    const int lane = (int)(threadIdx.x & 31);
    const int pj = lane % W;
    const int own = pj / L;
    const unsigned setMask = W >= 32 ? 0xffffffffu : (((1u << W) - 1u) << (lane - pj));
    const int N = p.env.shDegree;
    const double R = p.env.shR;
    FieldGeo g[K];
    Lanes<double, K> u, t;
    if constexpr (K == 1) {
        fieldGeo<W>(x, y, z, R, pj, g[0]);
    } else {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int src = lane - pj + k * L;
            fieldGeo<W>(__shfl_sync(setMask, x, src), __shfl_sync(setMask, y, src), __shfl_sync(setMask, z, src), R, pj,
                        g[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        u.set(k, g[k].u);
        t.set(k, g[k].t);
    }
    Lanes<T, K> uT, tT;
    if constexpr (kSplit) {
        uT = Lanes<T, K>::all(T(0));
        tT = uT;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            uT.set(k, g[k].u);
            tT.set(k, g[k].t);
        }
    }
    const int low = kSplit ? p.lowDeg : N;
    int at = 0;  // the block's first chunk
    for (int b = 0; b < tile.nblocks; ++b) {
        const int n64 = rowPairs64(b * W, N, low);
        Lanes<double, K> q, q1 = Lanes<double, K>::all(0.0), S[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) S[c] = Lanes<double, K>::all(0.0);
        double cL[K], sL[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            q.set(k, g[k].mag);
            cL[k] = g[k].cL;
            sL[k] = g[k].sL;
            g[k].cL = __fma_rn(g[k].cW, cL[k], -__dmul_rn(g[k].sW, sL[k]));
            g[k].sL = __fma_rn(g[k].cW, sL[k], __dmul_rn(g[k].sW, cL[k]));
            g[k].mag = __dmul_rn(g[k].mag, g[k].magW);
        }
        fieldRows<double, K, W, MODE, !kSplit>(tile, stream, pj, at, kSplit ? rowPairs64(b * W + pj, N, low) : n64, n64, u,
                                              t, q, q1, S);
        at += n64 * kChunks64 * W;
        if constexpr (kSplit) {
            Lanes<T, K> qT = Lanes<T, K>::all(T(0)), qT1 = qT, ST[6];
#pragma unroll
            for (int c = 0; c < 6; ++c) ST[c] = Lanes<T, K>::all(T(0));
#pragma unroll
            for (int k = 0; k < K; ++k) {
                qT.set(k, q.get(k));
                qT1.set(k, q1.get(k));
            }
            const int n32 = rowPairs32(b * W, N, low);
            fieldRows<T, K, W, MODE, true>(tile, stream, pj, at, n32, n32, uT, tT, qT, qT1, ST);
            at += n32 * kChunks32 * W;
#pragma unroll
            for (int c = 0; c < 6; ++c)
#pragma unroll
                for (int k = 0; k < K; ++k) S[c].v[k] = __dadd_rn(S[c].v[k], ST[c].get(k));
        }
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                g[k].acc[c] = __fma_rn(cL[k], S[2 * c].v[k], __fma_rn(sL[k], S[2 * c + 1].v[k], g[k].acc[c]));
    }
    if constexpr (MODE == TileRead::kStream) stream.rewind();
    // fold the set's partial sums of each object
#pragma unroll
    for (int off = W / 2; off > 0; off >>= 1)
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                g[k].acc[c] = __dadd_rn(g[k].acc[c], __shfl_xor_sync(setMask, g[k].acc[c], off));
    double a[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        a[c] = g[0].acc[c];
#pragma unroll
        for (int k = 1; k < K; ++k) a[c] = own == k ? g[k].acc[c] : a[c];
    }
    if (p.env.shTides) {
        double e[3];
        tidePart<L>(rec, pj % L, x, y, z, R, e);
#pragma unroll
        for (int off = L / 2; off > 0; off >>= 1)
#pragma unroll
            for (int c = 0; c < 3; ++c) e[c] = __dadd_rn(e[c], __shfl_xor_sync(setMask, e[c], off));
#pragma unroll
        for (int c = 0; c < 3; ++c) a[c] = __dadd_rn(a[c], e[c]);
    }
    const double inv = __drcp_rn(__dsqrt_rn(__fma_rn(z, z, __fma_rn(y, y, __dmul_rn(x, x)))));
    const double f = __dmul_rn(__ddiv_rn(p.env.shGM, R), inv);
#pragma unroll
    for (int c = 0; c < 3; ++c) out[c] = __dmul_rn(f, a[c]);
}

}  // namespace phop

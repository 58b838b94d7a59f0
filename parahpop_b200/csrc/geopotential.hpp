// Coefficient tile of the geopotential and its host-side construction.
//
// The acceleration of a spherical-harmonic field is itself a sum of solid
// harmonics, one degree and one order further: with the column functions
// p_nu,M = alpha^nu P_nu,M(sin phi) (alpha = R / r, fully normalised),
//     a_x = GM / R^2 alpha sum_M cos M lambda sum_nu Xc p + sin M lambda sum_nu Xs p
// and likewise a_y (Yc, Ys) and a_z (Zc, Zs), where row nu of column M holds
// constants formed here from C, S of degree n = nu - 1 and orders M - 1, M,
// M + 1 (Montenbruck & Gill, Satellite Orbits, 2000, section 3.2.5; the
// reference sums the same field term by term in spherical components,
// DegreeLoop.h:83-112).  One term is then one step of one recurrence and six
// sums, without latitude derivatives and without a division by cos phi.
//
// The recurrence p_{nu+1} = a alpha s p_nu - b alpha^2 p_{nu-1} is scaled
// per column (p = sigma q, sigma_{nu+1} = b sigma_{nu-1}) to
//     q_{nu+1} = A alpha s q_nu - alpha^2 q_{nu-1},
// so a row carries one recurrence factor A and six coefficients (x sigma).
// sigma_M = P_MM / cos^M phi, so a column starts from q_M = (alpha cos phi)^M.
//
// Layout: columns 0 .. order + 1 in blocks of W (W lanes, lane j takes column
// b W + j), rows in pairs; every lane of a block has the room of the block's
// longest column (zero rows past a column's end and for the lanes past the
// last column), so that a block's row loop can run uniformly.  A row pair of
// a lane is seven 16-byte chunks in FP64 (A0 A1 | Xc0 Xs0 | Yc0 Ys0 | Zc0 Zs0
// | Xc1 Xs1 | Yc1 Ys1 | Zc1 Zs1) and four in FP32 (A0 A1 Xc0 Xs0 | Yc0 Ys0
// Zc0 Zs0 | Xc1 Xs1 Yc1 Ys1 | Zc1 Zs1 - -), chunk c of pair i of lane j at
// ((i chunks + c) W + j): the lanes of a load read consecutive 16-byte words,
// and a block's pairs follow the block's before: the tile is one stream in
// the order the column loop reads it.  In split precision a block's FP64
// pairs come first, then its FP32 pairs; the rows of degrees n <= lowDeg +
// kLowMargin of a column are FP64, rounded up to whole pairs (by the column
// alone: the same rows whatever W).  The bytes are padded to whole stages of
// the stream (kStageChunks).
//
// kLowMargin: in this form the FP32 rounding of the row factors A is the same
// field error in every evaluation, and that of alpha sin phi and alpha^2 the
// same in every row of one, so the error of a day's orbit comes out larger
// than that of the spherical-component sums this form replaced although the
// error of one evaluation does not.  Split against FP64 after 24 h, mm, p99 /
// max, at low parts of 20 (degree 70) and 24 (degree 120): 10^4 LEO objects
// at degree 70, 10^5 of the uneven population, 10^5 LEO at degree 120
//     spherical components   1.93 / 6.41   0.74 / 6.31   1.64 / 8.29
//     margin 1               2.49 / 9.45   0.97 / 9.45   1.91 / 11.64
//     margin 9               1.37 / 6.08   0.55 / 5.57   1.15 / 6.97
//     margin 11              1.27 / 5.30   0.51 / 5.67   1.01 / 7.99
// The ten FP64 degrees beyond the first cost 7 % of the first run's time, 4 %
// of the second's and 6 % of the third's (nine FP64 degrees the same).  Two
// words for alpha sin phi and alpha^2 instead took 5, 11 and 11 % and left
// 1.80 / 6.94, 0.81 / 9.24 and 1.46 / 6.96.
#pragma once
#include <vector>

#if defined(__CUDACC__)
#define PHOP_GEO_HD __host__ __device__ __forceinline__
#else
#define PHOP_GEO_HD inline
#endif

namespace phop {

constexpr int kChunks64 = 7;  // 16-byte chunks of an FP64 row pair
constexpr int kChunks32 = 4;  // and of an FP32 row pair

constexpr int kLowMargin = 11;  // FP64 degrees beyond lowDeg: see above

// row nu of the last FP64 degree in a field of degree N whose FP64 low part
// is `lowDeg`
PHOP_GEO_HD int topRow64(int N, int lowDeg) { return (lowDeg + kLowMargin < N ? lowDeg + kLowMargin : N) + 1; }
// FP64 row pairs of column M (lowDeg >= N: all rows); they fall with M
PHOP_GEO_HD int rowPairs64(int M, int N, int lowDeg) {
    const int top = topRow64(N, lowDeg);
    const int rows = top - M + 1;
    return rows > 0 ? (rows + 1) / 2 : 0;
}
// FP32 row pairs that hold those of every column >= M
PHOP_GEO_HD int rowPairs32(int M, int N, int lowDeg) {
    const int top = topRow64(N, lowDeg);
    const int rows = N + 1 - (M <= top ? top : M - 1);
    return rows > 0 ? (rows + 1) / 2 : 0;
}

// Bytes of the first blocks of a tile that fit `limit`
inline int leadingBlocks(int nblocks, int W, int N, int lowDeg, int limit) {
    int bytes = 0;
    for (int b = 0; b < nblocks; ++b) {
        const int next = (rowPairs64(b * W, N, lowDeg) * kChunks64 + rowPairs32(b * W, N, lowDeg) * kChunks32) * W * 16;
        if (next > limit - bytes) break;
        bytes += next;
    }
    return bytes;
}

// A tile too large for shared memory is streamed through a ring of
// kRingStages stages per warp.
constexpr int kStageChunks = 128;  // 16-byte chunks of a stage: four a lane
constexpr int kRingStages = 8;
constexpr int kRingMirror = kChunks64 - 1;  // rows (W <= 8 chunks) repeated past the ring's end
constexpr int kRingBytes = (kRingStages * kStageChunks + kRingMirror * 8) * 16;

struct HostTile {
    std::vector<unsigned char> bytes;
    int nblocks = 0;
};

struct HostEnvironment;

// Tile for W lanes; split: rows above degree lowDeg in FP32.  The columns end
// at the last order that has a nonzero coefficient (plus one).
HostTile buildTile(const HostEnvironment& h, int W, bool split, int lowDeg);
// Last order with a nonzero coefficient.
int fieldOrder(const HostEnvironment& h);
// N_nm of the full normalisation (C = N_nm C_normalised).
double normFactor(int n, int m);

}  // namespace phop

// Host-side construction of the geopotential's coefficient tile (layout and
// formulas: geopotential.hpp).
#include "geopotential.hpp"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "engine.hpp"

namespace phop {

using real = long double;

// recurrence factors of the fully normalised Legendre functions, step to (n, m)
static real factorA(int n, int m) {
    return std::sqrt((real)(2 * n - 1) * (2 * n + 1) / ((real)(n - m) * (n + m)));
}
static real factorB(int n, int m) {
    return std::sqrt((real)(2 * n + 1) * (n + m - 1) * (n - m - 1) / ((real)(2 * n - 3) * (n + m) * (n - m)));
}

static real normFactorL(int n, int m) {
    real f = (m == 0 ? 1.0L : 2.0L) * (2 * n + 1);
    for (int k = n - m + 1; k <= n + m; ++k) f /= k;
    return std::sqrt(f);
}
double normFactor(int n, int m) { return (double)normFactorL(n, m); }

int fieldOrder(const HostEnvironment& h) {
    int last = 0;
    for (int n = 0; n <= h.shDegree; ++n)
        for (int m = last + 1; m <= std::min(n, h.shOrder); ++m) {
            const size_t t = (size_t)n * (n + 1) / 2 + m;
            if (h.shC[t] != 0.0 || h.shS[t] != 0.0) last = m;
        }
    return last;
}

namespace {
struct Row {
    double a = 0.0, x[6] = {0, 0, 0, 0, 0, 0};
};
}  // namespace

HostTile buildTile(const HostEnvironment& h, int W, bool split, int lowDeg) {
    HostTile out;
    if (!h.hasShape) {
        out.bytes.assign(kStageChunks * 16, 0);
        return out;
    }
    const int N = h.shDegree, order = fieldOrder(h);
    const int low = split ? lowDeg : N;
    const bool norm = h.shNormalized != 0;
    auto coef = [&](const std::vector<double>& t, int n, int m) -> real {
        if (m < 0 || m > n || m > order || n > N) return 0.0L;
        const real v = t[(size_t)n * (n + 1) / 2 + m];
        return norm || v == 0.0L ? v : v / normFactorL(n, m);
    };
    auto S = [&](int n, int m) -> real { return m > 0 ? coef(h.shS, n, m) : 0.0L; };
    // the rows of one column, nu = M .. N + 1
    auto column = [&](int M) {
        std::vector<Row> rows;
        std::vector<real> sigma(N + 3, 1.0L);
        real d = 1.0L;
        for (int k = 1; k <= M; ++k) d *= k == 1 ? std::sqrt(3.0L) : std::sqrt((2.0L * k + 1.0L) / (2.0L * k));
        for (int nu = M; nu <= N + 1; ++nu) {
            sigma[nu] = nu == M ? d : nu == M + 1 ? factorA(nu, M) * d : factorB(nu, M) * sigma[nu - 2];
            Row r;
            if (nu <= N) {
                const real next = nu == M ? factorA(nu + 1, M) * d : factorB(nu + 1, M) * sigma[nu - 1];
                r.a = (double)(factorA(nu + 1, M) * sigma[nu] / next);
            }
            const int n = nu - 1;
            if (n >= 0) {
                real x[6] = {0, 0, 0, 0, 0, 0};
                const real k = (real)(2 * n + 1) / (2 * n + 3);
                if (M >= 1) {  // from order m = M - 1
                    const int m = M - 1;
                    const real f = m == 0 ? std::sqrt(0.5L * k * (n + 2) * (n + 1))
                                          : 0.5L * std::sqrt(k * (n + m + 2) * (n + m + 1));
                    x[0] -= f * coef(h.shC, n, m);
                    x[1] -= f * S(n, m);
                    x[2] += f * S(n, m);
                    x[3] -= f * coef(h.shC, n, m);
                }
                if (M + 1 <= n) {  // from order m = M + 1
                    const int m = M + 1;
                    const real f = 0.5L * std::sqrt((m == 1 ? 2.0L : 1.0L) * k * (n - m + 2) * (n - m + 1));
                    x[0] += f * coef(h.shC, n, m);
                    x[1] += f * S(n, m);
                    x[2] += f * S(n, m);
                    x[3] -= f * coef(h.shC, n, m);
                }
                if (M <= n) {
                    const real f = std::sqrt(k * (n + M + 1) * (n - M + 1));
                    x[4] -= f * coef(h.shC, n, M);
                    x[5] -= f * S(n, M);
                }
                for (int c = 0; c < 6; ++c) r.x[c] = (double)(x[c] * sigma[nu]);
            }
            rows.push_back(r);
        }
        return rows;
    };
    const int columns = std::min(order, N) + 2;  // orders 0 .. order + 1
    out.nblocks = (columns + W - 1) / W;
    for (int b = 0; b < out.nblocks; ++b) {
        const int n64 = rowPairs64(b * W, N, low), n32 = rowPairs32(b * W, N, low);
        const size_t base = out.bytes.size();
        out.bytes.resize(base + ((size_t)n64 * kChunks64 + (size_t)n32 * kChunks32) * W * 16, 0);
        unsigned char* p64 = out.bytes.data() + base;
        unsigned char* p32 = p64 + (size_t)n64 * kChunks64 * W * 16;
        for (int j = 0; j < W; ++j) {
            const int M = b * W + j;
            if (M >= columns) break;
            const std::vector<Row> rows = column(M);
            auto at = [&](int i) { return i < (int)rows.size() ? rows[i] : Row{}; };
            const int own64 = rowPairs64(M, N, low);
            for (int i = 0; i < (split ? own64 : n64); ++i) {
                const Row r0 = at(2 * i), r1 = at(2 * i + 1);
                const double v[14] = {r0.a,    r1.a,    r0.x[0], r0.x[1], r0.x[2], r0.x[3], r0.x[4],
                                      r0.x[5], r1.x[0], r1.x[1], r1.x[2], r1.x[3], r1.x[4], r1.x[5]};
                for (int c = 0; c < kChunks64; ++c)
                    std::memcpy(p64 + (((size_t)i * kChunks64 + c) * W + j) * 16, v + 2 * c, 16);
            }
            for (int i = 0; i < n32; ++i) {
                const Row r0 = at(2 * own64 + 2 * i), r1 = at(2 * own64 + 2 * i + 1);
                const float v[16] = {(float)r0.a,    (float)r1.a,    (float)r0.x[0], (float)r0.x[1],
                                     (float)r0.x[2], (float)r0.x[3], (float)r0.x[4], (float)r0.x[5],
                                     (float)r1.x[0], (float)r1.x[1], (float)r1.x[2], (float)r1.x[3],
                                     (float)r1.x[4], (float)r1.x[5], 0.f,            0.f};
                for (int c = 0; c < kChunks32; ++c)
                    std::memcpy(p32 + (((size_t)i * kChunks32 + c) * W + j) * 16, v + 4 * c, 16);
            }
        }
    }
    const size_t stage = kStageChunks * 16;
    out.bytes.resize((out.bytes.size() + stage - 1) / stage * stage, 0);
    return out;
}

}  // namespace phop

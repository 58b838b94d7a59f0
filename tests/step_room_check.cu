// Host check of the step kernel's shared-memory split: for every compiled
// shape and fields of every degree up to 400, what the CTA holds by itself and
// what it asks for fit the 227 KiB a CTA may use.  Prints one JSON line.
#include <algorithm>
#include <cstdio>

#include "propagate.cuh"

using namespace phop;

static TileShape tileOf(int N, int W, bool split) {
    const int low = split ? (N > 80 ? kSplitFp64DegreeHigh : kSplitFp64Degree) : N, columns = N + 2;
    long b = 0;
    for (int k = 0; k < (columns + W - 1) / W; ++k)
        b += ((long)rowPairs64(k * W, N, low) * kChunks64 + (long)rowPairs32(k * W, N, low) * kChunks32) * W * 16;
    const int stage = kStageChunks * 16;
    return TileShape{(int)((b + stage - 1) / stage * stage), (columns + W - 1) / W, W, N, low};
}

int main() {
    const int kMax = 232448;
    int shapes = 0, over = 0, none = 0, most = 0;
    for (int split = 0; split < 2; ++split)
        for (int L = 1; L <= 16; L *= 2)
            for (int pair = 0; pair < 2; ++pair)
                for (int deep = 0; deep < 2; ++deep)
                    for (int duo = 0; duo < 2; ++duo) {
                        if ((pair && L > 4) || (deep && !hasDeepShape(L)) || (duo && !hasDuo(L, pair))) continue;
                        // the staging barrier, the mail and the quit words, in the 128-byte alignment of the dynamic part
                        const int mail = duo ? kDuoPairs * (32 / L) * (int)sizeof(DuoMail) + kDuoPairs * 4 : 0;
                        const int own = (8 + mail + 127) / 128 * 128;
                        const bool mayStream = duo ? L <= 4 : hasStream(L, deep);
                        for (int N = 1; N <= 400; ++N) {
                            const TileShape tile = tileOf(N, pair ? 2 * L : L, split != 0);
                            const int bound = stepThreadBound(L, deep, duo), halves = duo ? 2 : 1;
                            const StepRoom r = stepRoom(kMax, own, own, tile, L, duo != 0, bound, true, mayStream, hasPart(L, deep || duo));
                            const int threads = std::min(bound, r.threads);
                            const int dynamic = (r.stagedBytes > 0 ? r.stagedBytes : r.streamed ? threads / (32 * halves) * kRingBytes : 0)
                                                + kStageBytes * (threads / halves / L);
                            ++shapes;
                            over += own + dynamic > kMax || (r.stagedBytes > 0 && (r.streamed || r.stagedBytes > tile.bytes || r.stagedBytes % 16));
                            none += threads < 32 * halves;
                            most = std::max(most, own + dynamic);
                        }
                    }
    std::printf("{\"shapes\": %d, \"over\": %d, \"no_warp\": %d, \"most\": %d}\n", shapes, over, none, most);
    return 0;
}

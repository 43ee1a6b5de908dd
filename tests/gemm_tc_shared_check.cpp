// The shared memory of every tile, epilogue and tuning switch of the tensor-core
// products: each epilogue warp has its blocks, and all of it fits an SM.
#include "gemm_tc_shared.h"

#include <cstdio>

using namespace vitb200;

static int failures = 0;

static void check(bool ok, const char *what, int m, int n, int second, const TcForced &f,
                  const TcShared &s) {
    if (!ok) {
        ++failures;
        printf("%s: tile %d x %d, epilogue %d, stages=%d staging=%d ctas=%d: %d stages, "
               "%d bytes of staging, %d in all\n", what, m, n, second, f.stages, f.staging,
               f.ctas, s.stages, s.staging_bytes, s.bytes());
    }
}

int main() {
    const int tiles[][2] = {{128, 32}, {128, 64}, {128, 128}, {128, 256}, {256, 256}};
    for (const auto &tile : tiles) {
        const int m = tile[0], n = tile[1];
        for (int second = 0; second <= kGeluSlopeEight; ++second) {
            if ((second == kGeluSlopeEight && (m != 128 || n != 128)) ||
                (second >= kSecondResidual && m != 128)) {
                continue;   // not built
            }
            for (int stages = 0; stages <= kMaxStages + 1; ++stages) {
                for (int staging = 0; staging <= 2; ++staging) {
                    for (int ctas = 0; ctas <= 3; ++ctas) {
                        for (int options = 0; options < 4 * 12; ++options) {
                            TcForced forced;
                            forced.stages = stages;
                            forced.staging = staging;
                            forced.ctas = ctas;
                            const bool spread = n < 128 && (options & 1);
                            const TcShared s = tc_shared(m, n, second, 1 + options / 4,
                                                         options & 2, spread, forced);
                            check(s.staging_bytes >= tc_least_staging(m, n, second),
                                  "warps write past their staging", m, n, second, forced, s);
                            check(s.stages >= 1 && s.stages <= kMaxStages,
                                  "ring depth", m, n, second, forced, s);
                            check(s.bytes() <= kSmemLimit, "more than an SM has", m, n,
                                  second, forced, s);
                        }
                    }
                }
            }
            // Without switches: what the launches were measured with.
            const TcShared s = tc_shared(m, n, second, 12, false, false, TcForced());
            const bool slope = second >= kGeluSlope, pair = second == kSecondResidual;
            const int want_stages = n < 128              ? 4
                                    : n > 128            ? (m > 128 || slope ? 3 : 4)
                                    : (slope || pair)    ? 2 : 3;
            const int want_staging = (n <= 128 && !slope && !pair ? 16 : slope && n > 128
                                          ? 64 : 32) * 1024;
            check(s.stages == (n == 64 && want_staging == 32768 ? 3 : want_stages) &&
                      s.staging_bytes == want_staging, "default", m, n, second, TcForced(), s);
        }
    }
    printf("%d failures\n", failures);
    return failures != 0;
}

// The exponent spread's rounding (spread_x256 in f4j_split.cu) against integer
// arithmetic: random quotients, ones next to a half, exact halves, and the ends of
// the range.  Launches no kernel.
#include "../../flag4j_gb300/csrc/f4j_split.cu"
#include <cstdio>
#include <random>

int main() {
    long long bad = 0, tried = 0;
    std::mt19937_64 g(7);
    auto one = [&](long long num, long long cnt) {
        if (cnt < 1 || cnt > INT32_MAX || num < 1 || num >= cnt << 11) return;
        const long long want = (long long)(((__int128)512 * num + cnt) / (2 * cnt));
        tried++;
        if (spread_x256(num, (int)cnt) != want && ++bad < 5)
            printf("%lld / %lld: %d for %lld\n", num, cnt, spread_x256(num, (int)cnt), want);
    };
    one(57880, 7071);  // 2095.49 / 256
    for (int i = 0; i < 4000000; i++) {
        const long long cnt = 1 + (long long)(g() >> (33 + g() % 31));
        const long long q = (long long)(g() >> 45) % (2048 * 256);  // num / cnt near (q + 1/2) / 256
        one((long long)(g() % ((unsigned long long)cnt << 11)), cnt);
        const long long half = (long long)(((__int128)(2 * q + 1) * cnt) / 512);
        for (int d = -1; d <= 2; d++) one(half + d, cnt);
    }
    for (long long cnt : {1ll, 2ll, 3ll, 256ll, 8192ll, (long long)INT32_MAX})
        for (long long num : {1ll, cnt - 1, cnt, cnt + 1, (cnt << 11) - 1}) one(num, cnt);
    printf("%lld quotients, %lld wrong\n", tried, bad);
    return bad || tried < 4000000;
}

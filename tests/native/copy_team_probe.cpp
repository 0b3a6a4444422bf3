// Jobs of a CopyTeam: every slice is done once, none above the limit before it
// is raised, none of a dropped job after finish().  Prints the failures.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "host_copy.h"

int main(int argc, char** argv)
{
    const int workers = argc > 1 ? atoi(argv[1]) : 4, rounds = argc > 2 ? atoi(argv[2]) : 300;
    gahhg::CopyTeam team;
    const bool running = team.start(workers);
    long long bad = running != (workers > 0);
    for (int r = 0; r < rounds; r++) {
        const size_t n = (size_t)(r * 7 % 41), ring = 1 + (size_t)(r % 5);
        std::vector<std::atomic<int>> hits(n);
        std::atomic<size_t> limit{0};
        const int kind = r % 3;
        team.post(n, kind == 0 ? n : 0, [&](size_t i) {
            if (kind != 0 && i >= limit.load()) hits[i] += 100;
            hits[i]++;
        });
        if (kind == 0) {  // the caller helps
            while (team.help()) {
            }
            team.finish(false);
            for (size_t i = 0; i < n; i++) bad += hits[i] != 1 || !team.done(i);
        } else {
            const size_t stop = kind == 1 ? n : n / 2;  // kind 2: dropped half way
            for (size_t at = 0; at < stop;) {
                const size_t to = at + ring < stop ? at + ring : stop;
                limit = to;
                team.allow(to);
                for (; at < to; at++)
                    while (!team.done(at)) team.help();
            }
            team.finish(kind == 2);
            for (size_t i = 0; i < n; i++) bad += hits[i] != (i < stop ? 1 : 0);
        }
    }
    // copies of every alignment and remainder
    std::vector<unsigned char> a(4096), b(4096), c(4096);
    for (size_t i = 0; i < a.size(); i++) a[i] = (unsigned char)(i * 31 + 7);
    for (size_t to = 0; to < 17; to++)
        for (size_t from = 0; from < 9; from++)
            for (size_t n : {0, 1, 15, 16, 63, 64, 65, 1000, 2048}) {
                memset(b.data(), 0, b.size());
                memset(c.data(), 0, c.size());
                gahhg::copy_for_device(b.data() + to, a.data() + from, n);
                memcpy(c.data() + to, a.data() + from, n);
                bad += b != c;
            }
    printf("%lld\n", bad);
    return 0;
}

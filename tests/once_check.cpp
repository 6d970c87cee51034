// OncePerDevice: once on each device, again after an exception, and for eight threads at a
// time with nobody going on before it is done. Exits 1 on any difference.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <stdexcept>
#include <thread>
#include <vector>

#include "sph_once.hpp"

int main()
{
    sphgb::OncePerDevice once;
    int runs[2] = {0, 0};
    for (int k = 0; k < 3; ++k)
        for (int d = 0; d < 2; ++d) once(d, [&] { ++runs[d]; });
    bool ok = runs[0] == 1 && runs[1] == 1;

    int tries = 0;
    for (int k = 0; k < 3; ++k) {
        try {
            once(5, [&] {
                if (++tries == 1) throw std::runtime_error("refused");
            });
        } catch (const std::runtime_error &) {
            ok = ok && k == 0;
        }
    }
    ok = ok && tries == 2;

    std::atomic<int> done{0}, early{0}, count{0};
    std::vector<std::thread> ts;
    for (int t = 0; t < 8; ++t)
        ts.emplace_back([&] {
            once(7, [&] {
                ++count;
                std::this_thread::sleep_for(std::chrono::milliseconds(50));
                done = 1;
            });
            if (!done) ++early;
        });
    for (auto &t : ts) t.join();
    ok = ok && count == 1 && early == 0;
    std::printf("%s\n", ok ? "ok" : "differs");
    return ok ? 0 : 1;
}

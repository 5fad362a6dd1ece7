// OncePerDevice from several threads: a set-up runs before its pair counts as done, a failed one does not
// count, and no number of pairs is too many.  Built with -fsanitize=thread, which also reports any race.
#include <atomic>
#include <cstdio>
#include <thread>

#include "shflbw_internal.hpp"

int main() {
    constexpr int kPairs = 1000, kThreads = 8;
    static int set_up_again[kPairs];
    static std::atomic<int> calls[kPairs];
    static char kernels[kPairs / 8];
    shflbw::OncePerDevice table;
    std::atomic<int> bad{0};
    if (table.run(kernels, 0, [] { return SHFLBW_ERR_CUDA; }) != SHFLBW_ERR_CUDA) ++bad;
    auto work = [&] {
        for (int i = 0; i < kPairs; ++i)
            if (table.run(kernels + i / 8, i % 8, [&] { ++calls[i]; return SHFLBW_OK; }) != SHFLBW_OK || !calls[i].load()) ++bad;
    };
    std::thread t[kThreads];
    for (auto& th : t) th = std::thread(work);
    for (auto& th : t) th.join();
    for (int i = 0; i < kPairs; ++i) {
        const int before = calls[i];
        if (before < 1 || before > kThreads) ++bad;
        table.run(kernels + i / 8, i % 8, [&] { ++set_up_again[i]; return SHFLBW_OK; });
        if (set_up_again[i]) ++bad;                        // done already
    }
    std::printf("%s\n", bad ? "FAILED" : "ok");
    return bad ? 1 : 0;
}

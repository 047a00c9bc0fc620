// Handles in several threads whose launches of one kernel differ in shape.
//   two_handles_main lane|pool
// One thread solves large batches, three solve small ones (or the same on the
// pooled kernel with another CTA shape), each on a handle of its own.  Prints the
// calls that failed or whose lengths differ from the thread's first call, made
// before the others start.
#include <atomic>
#include <condition_variable>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <random>
#include <thread>
#include <vector>

#include "sbfs.h"

int main(int argc, char **argv)
{
    const bool pool = argc > 1 && !std::strcmp(argv[1], "pool");
    constexpr int kThreads = 4, kCalls = 3000, kN = 8;
    std::atomic<bool> stop{false};
    std::atomic<long> failed{0}, wrong{0}, calls{0};
    std::mutex mu;
    std::condition_variable cv;
    int ready = 0;
    auto work = [&](int id) {
        const bool first = id == 0;
        const int count = first ? (pool ? 20000 : 200000) : 40;
        sbfs_config cfg;
        sbfs_config_default(&cfg);
        if (pool) {
            cfg.small_kernel = 2;
            cfg.warps_per_cta = first ? 8 : 1;
        }
        sbfs_handle *h = nullptr;
        bool up = sbfs_create(&cfg, &h) == SBFS_OK;
        std::mt19937 rng(7 + id);
        std::vector<uint8_t> maps((size_t)count * 2 * kN);
        for (auto &x : maps) x = (uint8_t)(rng() % kN);
        std::vector<int32_t> ref(count), len(count);
        int64_t fv = 0;
        {
            std::unique_lock<std::mutex> lock(mu);   // the first calls one after another
            up = up && sbfs_verify_batch(h, maps.data(), kN, nullptr, kN, count, ref.data(), &fv, nullptr) == SBFS_OK;
            if (!up) ++failed;
            ++ready;
            cv.notify_all();
            cv.wait(lock, [&] { return ready == kThreads; });
        }
        for (int i = 0; up && (first ? i < kCalls : !stop.load()); ++i) {
            ++calls;
            if (sbfs_verify_batch(h, maps.data(), kN, nullptr, kN, count, len.data(), &fv, nullptr) != SBFS_OK) {
                if (failed++ < 3) std::printf("%s\n", sbfs_last_error(h));
            } else if (len != ref) {
                ++wrong;
            }
        }
        if (first) stop = true;
        sbfs_destroy(h);
    };
    std::vector<std::thread> t;
    for (int i = 0; i < kThreads; ++i) t.emplace_back(work, i);
    for (auto &x : t) x.join();
    std::printf("calls %ld failed %ld wrong %ld\n", calls.load(), failed.load(), wrong.load());
    return failed || wrong;
}

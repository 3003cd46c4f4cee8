// The selection heap's device code (fednl_heap.cuh) on the host, for schedules that a GPU seldom takes.
#include <algorithm>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <thread>

#define __device__
#define __forceinline__ inline
struct ulonglong2 {
    unsigned long long x, y;
};
using std::max;

#include "fednl_heap.cuh"

// The two warps of TopLEK's extraction, with the extracting one as late as it can be: after each meeting it
// goes on only when the other has reached the next one or has left.  Answers the steps at which they leave.
static int steps(int nch, int hit_at)
{
    int hit[2] = {0, 0};
    std::mutex mu;
    std::condition_variable cv;
    int met[2] = {0, 0};                 // meetings reached: extraction, windows
    bool left[2] = {false, false}, stuck = false;
    auto meet = [&](int me) {
        std::unique_lock<std::mutex> g(mu);
        const int n = ++met[me];
        cv.notify_all();
        cv.wait(g, [&] { return met[1 - me] >= n || left[1 - me]; });
        if (met[1 - me] < n) {           // the other left: this one would wait for ever
            stuck = true;
            return;
        }
        if (me == 0) cv.wait(g, [&] { return met[1] > n || left[1]; });
    };
    auto leave = [&](int me) {
        std::lock_guard<std::mutex> g(mu);
        left[me] = true;
        cv.notify_all();
    };
    std::thread a([&] {
        fednl::extract_steps(nch, hit, [](int) {}, [&] { meet(0); });
        leave(0);
    });
    std::thread b([&] {
        fednl::window_steps(nch, hit, true, [&](int q) { return q == hit_at; }, [&] {
            meet(1);
            if (stuck) hit[0] = hit[1] = 1;
        });
        leave(1);
    });
    a.join();
    b.join();
    std::printf("%d %d %d\n", met[0], met[1], stuck ? 1 : 0);
    return 0;
}

int main(int argc, char** argv)
{
    if (argc == 4 && !std::strcmp(argv[1], "steps")) return steps(std::atoi(argv[2]), std::atoi(argv[3]));
    return 2;
}

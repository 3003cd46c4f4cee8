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

// The lanes of a warp run one at a time, each from one __syncwarp() to the next before the following lane
// starts, in the given order or its reverse.
struct Warp {
    static constexpr int n = 32;
    std::mutex mu;
    std::condition_variable cv;
    bool reverse = false;
    int turn = 0, ended = 0;
    unsigned long long rounds[n] = {};
    bool done[n] = {};
    int at(int t) const { return reverse ? n - 1 - t : t; }
    void next()                          // with mu held: the next lane that still runs
    {
        do turn = (turn + 1) % n;
        while (done[at(turn)] && ended < n);
        cv.notify_all();
    }
    void start(int lane)
    {
        std::unique_lock<std::mutex> g(mu);
        cv.wait(g, [&] { return at(turn) == lane; });
    }
    void sync(int lane)
    {
        std::unique_lock<std::mutex> g(mu);
        ++rounds[lane];
        next();
        cv.wait(g, [&] { return at(turn) == lane; });
    }
    void end(int lane)
    {
        std::unique_lock<std::mutex> g(mu);
        done[lane] = true;
        ++ended;
        next();
    }
};
static Warp* g_warp;
static thread_local int g_lane;
static void __syncwarp() { g_warp->sync(g_lane); }

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

struct Heap {
    alignas(32) unsigned long long key_[4096];
    alignas(32) unsigned hid_[4096];
    fednl::HeapS h;
    Heap(int k, unsigned long long seed, int values)
    {
        h.key = key_ + 3;                // children 4i + 1 .. 4i + 4 on a 32-byte boundary
        h.hid = hid_ + 3;
        for (int i = 0; i < k; ++i) {
            seed = seed * 6364136223846793005ull + 1442695040888963407ull;
            h.key[i] = (seed >> 33) % values;
            h.hid[i] = (unsigned)i;
        }
        for (int i = (k - 2) / 4; i >= 0; --i) fednl::heap_sift(h, i, k);
    }
};

// `count` entries enter a heap of k by a warp and by one thread: the heaps and every lane's top must agree
static int lanes(int k, int count, int values, int reverse)
{
    Heap one(k, 7, values), all(k, 7, values);
    auto entry = [&](int t) { return (unsigned long long)((t * 2654435761u >> 8) % (3 * values)); };
    unsigned long long root = one.h.key[0];
    for (int t = 0; t < count; ++t)
        if (entry(t) > root) root = fednl::heap_replace_root(one.h, k, entry(t), (unsigned)(k + t));
    Warp w;
    w.reverse = reverse != 0;
    g_warp = &w;
    if (reverse) w.turn = 0;
    fednl::HeapMins mins;
    fednl::HeapTop top[Warp::n];
    std::thread th[Warp::n];
    for (int l = 0; l < Warp::n; ++l)
        th[l] = std::thread([&, l] {
            g_lane = l;
            w.start(l);
            top[l].load(all.h, &mins);
            for (int t = 0; t < count; ++t)
                if (entry(t) > top[l].K0 && top[l].root(entry(t), (unsigned)(k + t)))
                    top[l].below<true>(all.h, k, entry(t), (unsigned)(k + t));
            w.end(l);
        });
    for (auto& t : th) t.join();
    int bad = 0;
    for (int l = 1; l < Warp::n; ++l)
        bad += top[l].K0 != top[0].K0 || top[l].I0 != top[0].I0 || top[l].s1 != top[0].s1 || top[l].s2 != top[0].s2 ||
               top[l].s3 != top[0].s3 || top[l].s4 != top[0].s4 || top[l].t1 != top[0].t1 || top[l].t4 != top[0].t4;
    top[0].store(all.h);
    for (int i = 0; i < k; ++i) bad += one.h.key[i] != all.h.key[i] || one.h.hid[i] != all.h.hid[i];
    std::printf("%d %llu\n", bad, w.rounds[0]);
    return 0;
}

int main(int argc, char** argv)
{
    if (argc == 4 && !std::strcmp(argv[1], "steps")) return steps(std::atoi(argv[2]), std::atoi(argv[3]));
    if (argc == 6 && !std::strcmp(argv[1], "lanes"))
        return lanes(std::atoi(argv[2]), std::atoi(argv[3]), std::atoi(argv[4]), std::atoi(argv[5]));
    return 2;
}

// Buffers of threads (block_ipt_gb300/csrc/thread_slots.h): threads that follow
// one another share one, threads that run together have their own.  Built and
// run by tests/test_thread_slots.py.
#include <atomic>
#include <cstdio>
#include <set>
#include <thread>
#include <vector>

#include "thread_slots.h"

static std::atomic<int> made{0};

static double *make()
{
    ++made;
    return new double[4];
}

int main()
{
    using Slots = iptgb::ThreadSlots<double>;
    int bad = 0;
    for (int i = 0; i < 100; ++i) {
        std::thread t([&] { bad += Slots::mine(make) != Slots::mine(make); });
        t.join();
    }
    bad += made != 1;
    std::atomic<int> here{0};
    std::vector<double *> got(8);
    std::vector<std::thread> ts;
    for (int i = 0; i < 8; ++i) {
        ts.emplace_back([&, i] {
            got[i] = Slots::mine(make);
            ++here;
            while (here < 8) std::this_thread::yield();
        });
    }
    for (auto &t : ts) t.join();
    bad += std::set<double *>(got.begin(), got.end()).size() != 8;
    bad += made != 8;
    std::printf("made %d bad %d\n", (int)made, bad);
    return bad != 0;
}

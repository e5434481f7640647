// thread_slots.h - one small buffer per host thread that outlives the thread.
//
// A thread takes a buffer on its first use and hands it on when it ends, so
// there are as many as threads that ever held one at the same time.  No buffer
// is freed, and none made or freed while a thread ends: the threads' last
// moments are no place for calls into the CUDA runtime.
#pragma once

#include <mutex>
#include <vector>

namespace iptgb {

template <typename T>
class ThreadSlots {
public:
    // the calling thread's buffer; null where make() gives none
    static T *mine(T *(*make)())
    {
        thread_local Holder held;
        if (held.p == nullptr) {
            List &l = list();
            std::lock_guard<std::mutex> lock(l.mu);
            if (!l.free.empty()) {
                held.p = l.free.back();
                l.free.pop_back();
            }
        }
        if (held.p == nullptr) held.p = make();
        return held.p;
    }

private:
    struct List {
        std::mutex mu;
        std::vector<T *> free;
    };
    struct Holder {
        T *p = nullptr;
        ~Holder()
        {
            if (p == nullptr) return;
            List &l = list();
            std::lock_guard<std::mutex> lock(l.mu);
            l.free.push_back(p);
        }
    };
    // (never destroyed: threads may end after the statics)
    static List &list()
    {
        static List *l = new List;
        return *l;
    }
};

}  // namespace iptgb

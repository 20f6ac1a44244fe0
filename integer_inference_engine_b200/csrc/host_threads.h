// Host work shared among a few threads of one call.
#pragma once
#include <thread>
#include <utility>

namespace iie {

struct MakeThread {
    template <typename Work>
    std::thread operator()(Work &work) const { return std::thread([&work] { work(); }); }
};

// Runs `work`, which shares itself out and does not throw, on the calling thread and on up to `HELPERS` more.  Where the system gives no
// thread, those that there are do it all: nothing is thrown on, and every thread has ended when this returns.
template <int HELPERS, typename Work, typename Make = MakeThread>
void run_with_helpers(Work &&work, Make make = Make()) {
    std::thread helpers[HELPERS];
    try {
        for (auto &t : helpers) t = make(work);
    } catch (...) {}
    work();
    for (auto &t : helpers) if (t.joinable()) t.join();
}

}  // namespace iie

// run_with_helpers (csrc/host_threads.h) compiled for the CPU with a thread maker that fails at a given thread; see
// tests/test_host_threads_cpu.py.
#include <atomic>
#include <system_error>

#include "host_threads.h"

namespace {
struct FailingMaker {
    int left;
    template <typename Work>
    std::thread operator()(Work &work) {
        if (left-- <= 0) throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
        return iie::MakeThread()(work);
    }
};
}  // namespace

// pieces 0 .. n - 1 marked by three helpers of which `made` come to be; the number of threads that ran
extern "C" int h_share(int made, int n, int *marks) {
    std::atomic<int> next{0}, ran{0};
    auto work = [&]() {
        ran++;
        for (int i; (i = next.fetch_add(1)) < n;) marks[i]++;
    };
    iie::run_with_helpers<3>(work, FailingMaker{made});
    return ran;
}

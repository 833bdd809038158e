// Check of gpuvoxels_gb300/csrc/threads.h: every piece is done once, also where threads cannot be
// started or where some of them throw, and what they throw reaches the caller.  Exit status 0 when
// all hold.
#include "../gpuvoxels_gb300/csrc/threads.h"

#include <atomic>
#include <cstdio>
#include <new>

using gvx::run_threads;

int main() {
    int bad = 0;
    auto check = [&](bool ok, const char* what) {
        if (!ok) { std::printf("failed: %s\n", what); bad++; }
    };
    for (size_t most : {1, 2, 7, 1000}) {
        for (int limit : {0, 1, 3, 1000}) {   // threads the system starts
            std::atomic<int> next{0}, done{0};
            int started = 0;
            auto start = [&](auto&& f) {
                if (started >= limit) throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
                started++;
                return std::thread(f);
            };
            run_threads(most, [&]() { while (next++ < 500) done++; }, start);
            check(done == 500, "every piece done once");
            check(started <= limit && (size_t)started <= most - 1, "no more threads than asked for");
        }
        std::atomic<int> next{0}, done{0};
        bool got = false;
        try {
            run_threads(most, [&]() {
                for (int i = next++; i < 500; i = next++) {
                    if (i % 7 == 3) throw std::bad_alloc();
                    done++;
                }
            });
        } catch (const std::bad_alloc&) {
            got = true;
        }
        check(got, "what a thread throws reaches the caller");
    }
    return bad ? 1 : 0;
}

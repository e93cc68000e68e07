// The order of the server's admission (csrc/admission.h) on host threads: a
// job that waits for room is not passed by a later one that would fit, one
// with an earlier ticket goes first whenever it arrives, a job above the budget
// goes alone, and waiters return when the server stops.  Prints "faults M".
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

#include "admission.h"

namespace {

struct Bench {
    std::mutex mu;
    std::condition_variable cv;
    gsdr::Admission a;
    std::vector<std::thread> threads;
    std::map<int64_t, int> state;  // ticket: 1 admitted, -1 refused
    int faults = 0;

    explicit Bench(int64_t budget) { a.budget = budget; }
    ~Bench() {
        for (auto& t : threads) t.join();
    }
    // A job comes to step 1; returns once it is admitted or waits there.
    void come(int64_t ticket, int64_t bytes) {
        threads.emplace_back([this, ticket, bytes] {
            std::unique_lock<std::mutex> lock(mu);
            const bool ok = a.parse(lock, cv, ticket, bytes);
            state[ticket] = ok ? 1 : -1;
            cv.notify_all();
        });
        // (a job that begins to wait notifies nobody)
        std::unique_lock<std::mutex> lock(mu);
        for (int i = 0; i < 10000 && !state.count(ticket) && !a.is_waiting(ticket); i++)
            cv.wait_for(lock, std::chrono::milliseconds(1));
    }
    void leave(int64_t bytes) {
        std::lock_guard<std::mutex> lock(mu);
        a.release(bytes, false);
        cv.notify_all();
    }
    // The job's state; `want` is given 10 s to come true, any other 100 ms to
    // stay away.
    void expect(int64_t ticket, int want, const char* what) {
        std::unique_lock<std::mutex> lock(mu);
        auto now = [&] { return state.count(ticket) ? state[ticket] : 0; };
        if (want)
            cv.wait_for(lock, std::chrono::seconds(10), [&] { return now() == want; });
        else
            cv.wait_for(lock, std::chrono::milliseconds(100), [&] { return now() != 0; });
        if (now() != want) {
            std::printf("%s: job %lld is %d\n", what, (long long)ticket, now());
            faults++;
        }
    }
};

int waiting_job_is_not_passed() {
    Bench b(100);
    b.come(1, 60);
    b.expect(1, 1, "the first fits");
    b.come(2, 80);
    b.expect(2, 0, "no room beside the first");
    b.come(3, 30);  // fits beside the first
    b.expect(3, 0, "a later job that fits");
    b.leave(60);
    b.expect(2, 1, "the first has left");
    b.expect(3, 0, "no room beside the second");
    b.leave(80);
    b.expect(3, 1, "the second has left");
    return b.faults;
}

int earlier_ticket_first() {
    Bench b(100);
    b.come(1, 90);
    b.come(3, 60);
    b.come(2, 70);  // its slot is older, its count took longer
    b.expect(3, 0, "no room for the third");
    b.leave(90);
    b.expect(2, 1, "the earlier ticket");
    b.expect(3, 0, "the later ticket");
    b.leave(70);
    b.expect(3, 1, "room for the third");
    return b.faults;
}

int several_at_once_and_alone() {
    Bench b(100);
    b.come(1, 100);
    b.come(2, 40);
    b.come(3, 50);
    b.come(4, 300);
    b.come(5, 10);
    b.leave(100);
    b.expect(2, 1, "fits");
    b.expect(3, 1, "fits beside the second");
    b.expect(4, 0, "above the budget");
    b.expect(5, 0, "behind the fourth");
    b.leave(40);
    b.expect(4, 0, "the third still holds memory");
    b.leave(50);
    b.expect(4, 1, "alone");
    b.expect(5, 0, "beside a job above the budget");
    b.leave(300);
    b.expect(5, 1, "at last");
    return b.faults;
}

int stop_ends_the_waits() {
    Bench b(100);
    b.come(1, 100);
    b.come(2, 50);
    b.come(3, 50);
    {
        std::lock_guard<std::mutex> lock(b.mu);
        b.a.stopping = true;
        b.cv.notify_all();
    }
    b.expect(2, -1, "stopped");
    b.expect(3, -1, "stopped");
    return b.faults;
}

}  // namespace

int main() {
    const int faults = waiting_job_is_not_passed() + earlier_ticket_first() +
                       several_at_once_and_alone() + stop_ends_the_waits();
    std::printf("faults %d\n", faults);
    return faults != 0;
}

// admission.h -- the server's admission by device memory, in two steps
// (server.cu).  Host code without CUDA, so that its order is checked without a
// device (tests/admission_check.cpp).
//
// Step 1 reserves a job's parse buffers, step 2 its clustering footprint.  A
// job that does not fit waits until no other job holds memory (step 1) or
// clusters (step 2) and then goes alone.
//
// Step 1 is in the order of the tickets, which the scheduler gives out with the
// slots: while a job waits for room, no job with a later ticket reserves any,
// whether it would fit or not.  The jobs that hold memory then drain, so a
// large job waits for those in front of it and not for an endless run of
// smaller ones behind it.  (Jobs that have not come to step 1 yet, because their
// worker is still counting their records, are not waited for.)
#pragma once
#include <condition_variable>
#include <cstdint>
#include <mutex>

namespace gsdr {

// Every member is guarded by the mutex of the lock that the calls are given;
// cv is notified whenever another waiter may be able to go on.
struct Admission {
    int64_t budget = 0;
    int64_t used = 0;             // reserved bytes
    int holding = 0;              // jobs past step 1
    int clustering = 0;           // jobs past step 2
    bool stopping = false;        // waiters give up

    // Jobs waiting at step 1, one per slot at most: a list through the waiting
    // calls' own frames, so that waiting needs no memory.
    struct Waiter {
        int64_t ticket;
        Waiter* next;
    };
    Waiter* waiting = nullptr;

    bool is_waiting(int64_t ticket) const {
        for (const Waiter* w = waiting; w; w = w->next)
            if (w->ticket == ticket) return true;
        return false;
    }
    bool is_first(int64_t ticket) const {
        for (const Waiter* w = waiting; w; w = w->next)
            if (w->ticket < ticket) return false;
        return true;
    }

    // False when the server stops.
    bool parse(std::unique_lock<std::mutex>& lock, std::condition_variable& cv, int64_t ticket,
               int64_t bytes) {
        Waiter me{ticket, waiting};
        waiting = &me;
        cv.wait(lock, [&] {
            return stopping || (is_first(ticket) && (used + bytes <= budget || holding == 0));
        });
        Waiter** at = &waiting;
        while (*at != &me) at = &(*at)->next;
        *at = me.next;
        cv.notify_all();  // the next ticket may fit as well
        if (stopping) return false;
        used += bytes;
        holding++;
        return true;
    }

    bool cluster(std::unique_lock<std::mutex>& lock, std::condition_variable& cv, int64_t bytes) {
        cv.wait(lock, [&] { return stopping || used + bytes <= budget || clustering == 0; });
        if (stopping) return false;
        used += bytes;
        clustering++;
        return true;
    }

    // A job past step 1 (and step 2: clustered) gives its reservations back.
    // The caller notifies.
    void release(int64_t bytes, bool clustered) {
        used -= bytes;
        holding--;
        if (clustered) clustering--;
    }
};

}  // namespace gsdr

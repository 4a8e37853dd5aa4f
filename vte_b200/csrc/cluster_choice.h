// Which clusters, if any, serve a call of vteb_split_kv_decode, and the record of what has been decided.  Plain C++: what
// asks the device comes in as functions.
#pragma once

#include <pthread.h>

struct ClusterCall {
    int device, num_q_heads, num_kv_heads, head_dim, batch, num_sms;
    long long context;
    bool operator==(const ClusterCall& o) const {
        return device == o.device && num_q_heads == o.num_q_heads && num_kv_heads == o.num_kv_heads && head_dim == o.head_dim &&
               batch == o.batch && num_sms == o.num_sms && context == o.context;
    }
};
struct ClusterChoice { int kind, parts; };            // parts 0: no clusters

// The last 64 decisions.  Sizes and the device alone decide; the device is part of the key because what lets a kernel run
// there (shared memory, cluster size) is set, for each device, by the queries that the first decision makes.
class ClusterChoices {
public:
    // `estimate(kind, parts, resident)`: microseconds, negative where the kernels do not cover the geometry.
    // `never_slower(kind, parts, resident)`: whether that holds whatever the lengths are, which the host does not see here.
    // `resident(kind, parts, &n)`: readies the kernel on the device and says how many clusters run at once; false where
    // that cannot be had, and then another answer serves the call and nothing is recorded.
    template <class Estimate, class NeverSlower, class Resident>
    ClusterChoice choose(const ClusterCall& call, double below, Estimate estimate, NeverSlower never_slower, Resident resident) {
        ClusterChoice best = {0, 0};
        bool found = false;
        pthread_mutex_lock(&lock_);
        for (unsigned i = 0; i < count_ && i < kKept && !found; ++i)
            if ((found = known_[i].call == call)) best = known_[i].choice;
        pthread_mutex_unlock(&lock_);
        if (found) return best;
        static const int kParts[] = {2, 3, 4, 5, 6, 8, 9, 12, 16};
        bool all_answered = true;
        for (int kind = 1; kind <= 2; ++kind)
            for (int parts : kParts) {
                const double least = estimate(kind, parts, call.batch * call.num_kv_heads);      // with room for all clusters at once
                if (least < 0.0 || least >= below) continue;
                int n = 0;
                if (!resident(kind, parts, &n)) { all_answered = false; continue; }
                const double us = n > 0 ? estimate(kind, parts, n) : below;
                if (us < below && never_slower(kind, parts, n)) { below = us; best.kind = kind; best.parts = parts; }
            }
        if (all_answered) {
            pthread_mutex_lock(&lock_);
            known_[count_ % kKept] = {call, best};
            if (++count_ == 2 * kKept) count_ = kKept;
            pthread_mutex_unlock(&lock_);
        }
        return best;
    }

private:
    static constexpr unsigned kKept = 64;
    struct Entry { ClusterCall call; ClusterChoice choice; };
    pthread_mutex_t lock_ = PTHREAD_MUTEX_INITIALIZER;
    Entry known_[kKept];
    unsigned count_ = 0;
};

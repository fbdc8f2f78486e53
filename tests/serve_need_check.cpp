// CPU check of the serving loop's admission (serve_sched.h) under scratch
// needs that do not rise with the reads of a launch: whatever the steps of
// need() from min_batch reads on, an admitted request is launched in pieces until it is done, no
// launch takes more than the pool holds, and none but a request's last is
// shorter than min_batch.  Exits 0 when every check holds.
#include <cstdio>
#include <cstdlib>

#include "../esperanto_gb300/csrc/serve_sched.h"

static void check(bool ok, const char *what) {
    if (ok) return;
    std::fprintf(stderr, "failed: %s\n", what);
    std::exit(1);
}

// Runs the jobs to their end, one launch at a time; returns the launches.
static int drain(serve::Scheduler &s, std::vector<serve::Job> &jobs, uint64_t min_batch) {
    for (auto &j : jobs) {
        check(s.admissible(j), "admissible");
        s.push(&j);
    }
    int launches = 0;
    std::vector<serve::Job *> done;
    while (!s.empty()) {
        serve::Launch L;
        check(s.next(L), "an idle pool always takes an admitted request");
        check(L.bytes <= s.pool().size(), "within the pool");
        bool last = false;
        for (auto &p : L.pieces) last |= p.job->next == p.job->n;
        check(L.n >= min_batch || last, "no short launch");
        s.finish(L, done);
        check(++launches < 100000, "ends");
    }
    check(done.size() == jobs.size(), "every job is done");
    for (auto &j : jobs) check(j.done == j.n, "every read is done");
    return launches;
}

int main() {
    {  // up to 1,040 reads and 1,400 to 1,500 fit
        auto need = [](uint64_t n, uint32_t, uint32_t) -> uint64_t {
            return n <= 1040 || (n >= 1400 && n <= 1500) ? 1000 : 5000;
        };
        serve::Scheduler s(1024, 8192, 1024, need);
        std::vector<serve::Job> jobs(1);
        jobs[0].n = 3 * 1024;
        drain(s, jobs, 1024);
    }
    {  // falling with the size of the reads, and with steps in n
        auto need = [](uint64_t n, uint32_t m, uint32_t) -> uint64_t {
            const uint64_t step = n < 2000 ? 700 : (n < 40000 ? 300 : 1500);
            return n * step / (m > 100 ? 3 : 1);
        };
        for (uint64_t pool : {1ull << 20, 6ull << 20, 40ull << 20}) {
            serve::Scheduler s(pool, 131072, 1024, need);
            std::vector<serve::Job> jobs(40);
            uint32_t x = 1;
            for (auto &j : jobs) {
                x = x * 1664525u + 1013904223u;
                j.n = 1 + x % 90000;
                j.max_m = j.max_n = x >> 16 & 1 ? 150 : 50;
            }
            drain(s, jobs, 1024);
            check(s.pool().used() == 0, "all scratch returned");
        }
    }
    std::puts("ok");
    return 0;
}

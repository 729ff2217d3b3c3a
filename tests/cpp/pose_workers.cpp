// The host worker threads of rf_epipolar.cpp, one situation per run (argv[1]);
// exits 0 when it went as it should, 1 with a line on stderr otherwise.
#include "rf_epipolar.cpp"

#include <chrono>
#include <cstdio>
#include <string>

#include <sched.h>
#include <signal.h>
#include <sys/wait.h>

using namespace rf_epi;

namespace {

int fail(const char* what) {
    std::fprintf(stderr, "%s\n", what);
    return 1;
}

// every index of a loop exactly once
bool loop_runs(int n) {
    std::vector<std::atomic<int>> seen(n);
    parallel_for(n, [&](int i) { seen[i]++; });
    return std::all_of(seen.begin(), seen.end(), [](const std::atomic<int>& s) { return s == 1; });
}

// the exit status of a forked child that runs `f`, or -1 if it takes over 10 s
template <class F>
int child(F&& f) {
    const pid_t pid = fork();
    if (pid == 0) _exit(f());
    for (int ms = 0; ms < 10000; ms += 5) {
        int st = 0;
        if (waitpid(pid, &st, WNOHANG) == pid) return WIFEXITED(st) ? WEXITSTATUS(st) : -2;
        std::this_thread::sleep_for(std::chrono::milliseconds(5));
    }
    kill(pid, SIGKILL);
    waitpid(pid, nullptr, 0);
    return -1;
}

// a child of a process that holds the workers: lets go of them, has loops run, holds
// workers of its own
int forked() {
    hold_workers();
    if (!loop_runs(200)) return fail("parent's loop");
    std::this_thread::sleep_for(std::chrono::milliseconds(50));  // the workers wait
    const int st = child([] {
        if (!loop_runs(200)) return 2;
        release_workers();
        if (!loop_runs(200)) return 3;
        hold_workers();
        if (!loop_runs(200)) return 4;
        release_workers();
        return 0;
    });
    if (st != 0) return fail(st == -1 ? "the child hangs" : "the child's loop");
    if (!loop_runs(200)) return fail("parent's loop after the fork");
    release_workers();
    return 0;
}

// the same while another thread holds and lets go, so that the fork may fall into it
int forked_busy() {
    std::atomic<bool> stop{false};
    std::thread other([&] {
        while (!stop) {
            hold_workers();
            release_workers();
        }
    });
    int st = 0;
    for (int i = 0; i < 40 && st == 0; i++)
        st = child([] {
            if (!loop_runs(200)) return 2;
            hold_workers();
            if (!loop_runs(200)) return 3;
            release_workers();
            return 0;
        });
    stop = true;
    other.join();
    return st == 0 ? 0 : fail(st == -1 ? "the child hangs" : "the child's loop");
}

// a loop whose body throws, in the caller's share and in the workers', with other
// callers' loops running beside it
int throwing() {
    hold_workers();
    std::atomic<bool> stop{false}, bad{false};
    std::thread other([&] {
        while (!stop)
            if (!loop_runs(64)) bad = true;
    });
    for (int k = 0; k < 500; k++) {
        bool caught = false;
        try {
            parallel_for(64, [&](int i) {
                if (i % 8 == k % 8) throw std::bad_alloc();
            });
        } catch (const std::bad_alloc&) {
            caught = true;
        }
        if (!caught) return fail("the exception is lost");
        if (!loop_runs(64)) return fail("the loop after it");
    }
    stop = true;
    other.join();
    release_workers();
    return bad ? fail("another caller's loop") : 0;
}

// a handle made by a thread bound to one CPU: the loops of a thread that is not run
// where that one may run (and the other way round)
int affinity() {
    cpu_set_t all, one;
    CPU_ZERO(&all);
    if (sched_getaffinity(0, sizeof all, &all) != 0) return fail("sched_getaffinity");
    CPU_ZERO(&one);
    for (int c = 0; c < CPU_SETSIZE && CPU_COUNT(&one) == 0; c++)
        if (CPU_ISSET(c, &all)) CPU_SET(c, &one);
    if (CPU_EQUAL(&one, &all)) return 0;  // a single CPU: nothing to tell apart
    for (int k = 0; k < 2; k++) {
        const cpu_set_t *maker = k ? &all : &one, *caller = k ? &one : &all;
        sched_setaffinity(0, sizeof *maker, maker);
        hold_workers();
        sched_setaffinity(0, sizeof *caller, caller);
        std::atomic<int> elsewhere{0};
        for (int r = 0; r < 20; r++)
            parallel_for(256, [&](int) {
                cpu_set_t mine;
                CPU_ZERO(&mine);
                sched_getaffinity(0, sizeof mine, &mine);
                if (!CPU_EQUAL(&mine, caller)) elsewhere++;
                std::this_thread::sleep_for(std::chrono::microseconds(20));
            });
        release_workers();
        if (elsewhere) return fail(k ? "on other CPUs than the caller's" : "bound to the maker's CPU");
    }
    return 0;
}

}  // namespace

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "forked") return forked();
    if (what == "forked_busy") return forked_busy();
    if (what == "throwing") return throwing();
    if (what == "affinity") return affinity();
    return fail("unknown situation");
}

// Host-side check of fork_scope.h with a context that only counts: every way
// out of the scope orders the context's stream after the side streams, once,
// and nothing throws while an exception unwinds.
#include <cstdio>
#include <stdexcept>

#include "fork_scope.h"

struct Fake {
    int forks = 0, joins = 0, drains = 0, n = 0;
    bool fork_fails = false, join_fails = false;
    void fork(int k) {
        if (fork_fails) throw std::runtime_error("fork");
        ++forks;
        n = k;
    }
    void join(int k) {
        if (join_fails) throw std::runtime_error("join");
        ++joins;
        n = k;
    }
    void drain(int k) noexcept {
        ++drains;
        n = k;
    }
};

int fails = 0;
void expect(const char* what, bool ok) {
    if (!ok) {
        std::printf("fail %s\n", what);
        ++fails;
    }
}

// the scope with a launch that may fail; whether an exception came out
bool run(Fake& f, int n, bool launch_fails) {
    try {
        hmb::ForkScope<Fake> scope(f, n);
        if (launch_fails) throw std::runtime_error("launch");
        scope.join();
    } catch (const std::runtime_error&) {
        return true;
    }
    return false;
}

int main() {
    Fake a;
    expect("plain", !run(a, 2, false) && a.forks == 1 && a.joins == 1 && a.drains == 0 && a.n == 2);
    Fake b;
    expect("launch fails", run(b, 2, true) && b.joins == 0 && b.drains == 1 && b.n == 2);
    Fake c;
    c.join_fails = true;
    expect("join fails", run(c, 3, false) && c.drains == 1 && c.n == 3);
    Fake d;
    d.fork_fails = true;
    expect("fork fails", run(d, 1, false) && d.joins == 0 && d.drains == 0);
    Fake e;
    expect("no side stream", !run(e, 0, false) && !e.forks && !e.joins && !e.drains);
    Fake g;
    expect("no side stream, launch fails", run(g, 0, true) && !g.joins && !g.drains);
    if (fails) return 1;
    std::printf("ok\n");
    return 0;
}

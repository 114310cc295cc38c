"""Forks and joins of a step graph (csrc/branch.hpp) against a fake of the
runtime's calls: whichever of them fails, nothing is issued to a stream that
is outside the capture, the failure is reported, and streams and events are
created all or not at all."""
import subprocess
from pathlib import Path

REPO = Path(__file__).resolve().parent.parent

HARNESS = r"""
#include <cstdio>
#include "branch.hpp"
using namespace fipi;

// streams and events are small numbers, 0 = none; stream 1 is being captured
struct Fake {
    int fail_at = 0, calls = 0, alive = 0, next = 2;
    bool captured[16] = {}, marked[16] = {};  // streams in the capture; events recorded in it
    int next_error() { return ++calls == fail_at ? 700 : 0; }
    int make(int* x) {
        if (int e = next_error()) { *x = 15; return e; }  // garbage with the error
        ++alive;
        *x = next++;
        return 0;
    }
    int stream(int* s) { return make(s); }
    int event(int* e) { return make(e); }
    int record(int e, int s) {
        if (int err = next_error()) return err;
        marked[e] = captured[s];
        return 0;
    }
    int wait(int s, int e) {
        if (int err = next_error()) return err;
        if (marked[e]) captured[s] = true;
        return 0;
    }
    void drop(int) { --alive; }
};

int main() {
    int bad = 0;
    for (int fail = 0; fail <= 8; ++fail) {  // the eight calls of a step with two branches
        Fake rt;
        int main_stream = 1, side = 2;
        BranchEvents<int> ev;
        ev.fork[0] = 3; ev.fork[1] = 4; ev.join[0] = 5; ev.join[1] = 6;
        rt.captured[1] = true;
        rt.fail_at = fail;
        int issued = 0, outside = 0;
        auto work = [&] { ++issued; outside += !rt.captured[main_stream]; };
        StepBranches<Fake, int, int> br{rt, main_stream, side, ev};
        br.fork(0, work); work(); br.join(0);
        br.fork(1, work); work(); br.join(1);
        if (issued != 4 || outside || main_stream != 1 || side != 2 || (br.err != 0) != (fail != 0)) {
            std::printf("step, call %d: issued %d, outside the capture %d, error %d\n", fail, issued, outside, br.err);
            bad = 1;
        }
    }
    for (int fail = 0; fail <= 5; ++fail) {  // one stream, four events
        Fake rt;
        rt.fail_at = fail;
        int side = 0;
        BranchEvents<int> ev;
        const int e = make_branches(rt, side, ev);
        const bool all = side && ev.fork[0] && ev.fork[1] && ev.join[0] && ev.join[1];
        const bool none = !side && !ev.fork[0] && !ev.fork[1] && !ev.join[0] && !ev.join[1];
        if ((e != 0) != (fail != 0) || !(e ? none && rt.alive == 0 : all && rt.alive == 5)) {
            std::printf("create, call %d: error %d, alive %d\n", fail, e, rt.alive);
            bad = 1;
        }
        drop_branches(rt, side, ev);
        if (rt.alive) bad = 1;
    }
    return bad;
}
"""


def test_every_failing_call_is_seen(tmp_path):
    src, exe = tmp_path / "h.cpp", tmp_path / "h"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(REPO / "fipi_gb300/csrc"), str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout

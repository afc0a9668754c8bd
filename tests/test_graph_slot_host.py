"""Which captured graph an evaluation launches (csrc/graph_slot.h), compiled
with the host compiler and a capture that fails on command: a graph captured
for another state is never launched, whatever becomes of the new capture, and a
later capture that works is used again."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "graph_slot.h"
#include <cstdio>
struct Graph { int state; };
int main() {
    Graph* exec = nullptr;
    int destroyed = 0, captures = 0;
    // evaluation of `state`, whose capture works or not; `keep`: the failing
    // capture leaves the old executable where it is. Prints what is launched.
    auto evaluate = [&](int state, bool works, bool keep) {
        const bool stale = !exec || exec->state != state;
        const bool go = amg::launchable(exec, stale, [&] {
            captures++;
            if (works) {
                delete exec;
                exec = new Graph{state};
            } else if (!keep) {
                delete exec;
                exec = nullptr;
            }
            return works;
        }, [&](Graph* g) { destroyed++; delete g; });
        if (go != (exec != nullptr)) std::printf("inconsistent ");
        std::printf("%d ", go ? exec->state : -1);
    };
    evaluate(1, true, true);    // first capture
    evaluate(1, true, true);    // launched again without one
    evaluate(2, false, true);   // new state, its capture fails: not the graph of state 1
    evaluate(2, false, true);   // tried again
    evaluate(2, true, true);    // works now
    evaluate(3, false, false);  // fails with the old one already gone
    evaluate(3, true, true);
    std::printf("captures %d destroyed %d\n", captures, destroyed);
}
"""


def test_a_stale_graph_is_never_launched(tmp_path):
    src = tmp_path / "slot.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "slot")
    subprocess.check_call(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "polmdqc_b200", "csrc"),
                           str(src), "-o", exe])
    assert subprocess.check_output([exe], text=True).strip() == "1 1 -1 -1 2 -1 3 captures 6 destroyed 1"

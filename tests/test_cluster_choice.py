"""The record of which clusters serve a call of the direct entry point (csrc/cluster_choice.h), compiled for the CPU with
functions that stand for the device."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "vte_b200" / "csrc"

HARNESS = r"""
#include <cstdio>
#include "cluster_choice.h"

static int queries = 0, failing = 0, slower_up_to = 0;
static ClusterChoice ask(ClusterChoices& c, int device, long long context) {
    const ClusterCall call = {device, 12, 2, 128, 4, 148, context};
    return c.choose(call, 10.0,
        [&](int kind, int parts, int resident) { return kind == 2 && parts == 16 ? -1.0 : resident < 8 ? 50.0 : 12.0 / parts + kind; },
        [&](int kind, int parts, int resident) { return parts > slower_up_to && resident > 0; },
        [&](int kind, int parts, int* n) { ++queries; *n = parts > 9 ? 4 : 16; return !(failing == 1 || (failing == 2 && parts == 9)); });
}
#define SAY(x) std::printf("%s %d\n", #x, (int)(x))
int main() {
    ClusterChoices c;
    const ClusterChoice first = ask(c, 0, 4096);
    SAY(first.kind); SAY(first.parts);                      // 1 and 9: the largest of which all eight pairs fit
    int before = queries;
    ask(c, 0, 4096); SAY(queries - before);                 // known
    ask(c, 1, 4096); SAY(queries - before > 0);             // another device of the same size: asked, and made ready
    failing = 2; SAY(ask(c, 0, 5000).parts);                // one answer missing: the next best
    failing = 1; SAY(ask(c, 0, 5000).parts);                // none to be had
    failing = 0; SAY(ask(c, 0, 5000).parts);                // neither was recorded
    slower_up_to = 8; SAY(ask(c, 2, 4096).parts);           // what a skewed batch could make slower is passed over,
    slower_up_to = 9; SAY(ask(c, 2, 5000).parts);           // down to no clusters at all
    slower_up_to = 0;
    for (int i = 0; i < 1000; ++i) ask(c, 0, 6000 + i);
    before = queries; ask(c, 0, 6999); SAY(queries - before);        // the last is known,
    ask(c, 0, 4096); SAY(queries - before > 0);                      // the first of a thousand not any more
    return 0;
}
"""


@pytest.fixture(scope="module")
def said(tmp_path_factory):
    d = tmp_path_factory.mktemp("cluster_choice")
    (d / "harness.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", "-o", str(d / "harness"), str(d / "harness.cpp")], check=True)
    return [line.split()[-1] for line in subprocess.run([str(d / "harness")], check=True, capture_output=True, text=True).stdout.splitlines()]


def test_choices_are_kept_for_each_device_and_only_when_every_candidate_answered(said):
    assert said == ["1", "9", "0", "1", "8", "0", "9", "9", "0", "0", "1"]

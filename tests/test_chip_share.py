"""How many SMs and lanes a verify launch plans with while other calls are at work on the
same device (csrc/chip_share.h), on the CPU: a lone call has the whole chip, calls side by
side do not plan with more than there is, and nothing stays counted."""
import os
import random
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "icp-gpu_b200", "csrc")
SMS = 148

DRIVER = r"""
#include <cstdio>
#include <iostream>
#include <string>
#include "chip_share.h"
// one command a line: b use device (B: a server's) | p use n expect -> lanes | s use need expect -> share |
// h use sms | w use (ends when its flag is up) | f use (its flag) | e use
int main() {
    static bls::ChipUse uses[8];
    static bool flag[8];
    std::string op;
    int u, a, x;
    while (std::cin >> op >> u) {
        if (op == "b" || op == "B") { std::cin >> a; flag[u] = false; uses[u].begin(a, 148, op == "b"); }
        if (op == "p") { std::cin >> a >> x; std::cout << uses[u].plan_verify(a, x != 0) << "\n"; }
        if (op == "s") { std::cin >> a >> x; std::cout << uses[u].share(a, x != 0) << "\n"; }
        if (op == "h") { std::cin >> a; uses[u].hold(a); }
        if (op == "w") uses[u].end_when([](const void* f) { return *static_cast<const bool*>(f); }, &flag[u]);
        if (op == "f") flag[u] = true;
        if (op == "e") uses[u].end();
    }
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("share")
    (d / "driver.cpp").write_text(DRIVER)
    exe = str(d / "driver")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, str(d / "driver.cpp"), "-o", exe,
                           "-lpthread"])

    def run(script):
        out = subprocess.run([exe], input="\n".join(script), text=True, capture_output=True, check=True)
        return [int(v) for v in out.stdout.split()]
    return run


def held(n, lanes):
    return SMS if n > 32 * SMS else min(SMS, -(-n * lanes // 32))


@pytest.mark.parametrize("n,lanes", [(1, 4), (8 * SMS, 4), (8 * SMS + 1, 2), (16 * SMS, 2), (16 * SMS + 1, 1),
                                     (32 * SMS, 1), (32 * SMS + 1, 4), (40 * SMS + 1, 2), (48 * SMS + 1, 1)])
def test_a_lone_call_has_the_whole_chip(plan, n, lanes):
    again = ["b 0 0", f"p 0 {n} 1", "e 0"] * 3
    assert plan(again) == [lanes] * 3
    assert plan(["b 0 0", f"p 0 {n} 0", "w 0", "f 0"] * 3) == [lanes] * 3


@pytest.mark.parametrize("n,calls", [(8 * SMS, 2), (8 * SMS, 3), (16 * SMS, 2), (300, 4), (37 * 32, 4), (1, 8)])
def test_calls_that_begin_together_fit_side_by_side(plan, n, calls):
    got = plan([f"b {c} 0" for c in range(calls)] + [f"p {c} {n} 1" for c in range(calls)])
    assert sum(held(n, lanes) for lanes in got) <= SMS


def test_a_batch_beside_a_large_one_takes_what_is_free(plan):
    # 4,096 items hold 128 SMs: 500 items fit the other twenty with a lane each
    assert plan(["b 0 0", "p 0 4096 1", "b 1 0", "p 1 500 1"]) == [1, 1]
    assert plan(["b 0 0", "p 0 4096 1", "b 1 0", "p 1 150 1"]) == [1, 4]
    # no room at all: it waits in any case, and plans with half the chip
    assert plan(["b 0 0", f"p 0 {32 * SMS} 1", "b 1 0", f"p 1 {8 * SMS} 1"]) == [1, 2]
    # a small launch keeps its 4 SMs, and the two large ones part the rest
    assert plan(["b 0 0", "p 0 1000 0", "b 1 0", "p 1 32 0", "b 2 0", "p 2 1000 0", "b 3 0", "s 3 148 0"]) == [4, 4, 2, 48]


def test_calls_that_return_early_are_expected_again(plan):
    """three contexts whose launches only show up one by one: after the first time each
    leaves the others their part; alone again, a context has the chip from the second call"""
    burst = [line for c in range(3) for line in (f"b {c} 0", f"p {c} {8 * SMS} 1", f"w {c}")] + ["f 0", "f 1", "f 2"]
    got = plan(burst * 3 + ["b 0 0", f"p 0 {8 * SMS} 1", "e 0"] * 2)
    for k in (1, 2):
        assert sum(held(8 * SMS, lanes) for lanes in got[3 * k:3 * k + 3]) <= SMS
    assert got[-1] == 4


def test_a_server_knows_its_own_queue(plan):
    """slots: the first requests of a burst, then the bulk, which no one follows"""
    first = ["B 0 0", "p 0 10 0", "B 1 0", "p 1 20 0", "B 2 0", "p 2 1000 0"]
    done = ["e 0", "e 1", "e 2"]
    assert plan(first + done + first) == [4, 4, 4] * 2
    # and does not make a context that calls alone afterwards, or beside it, hold back
    assert plan((first + done + ["b 3 0", f"p 3 {8 * SMS} 1", "e 3"]) * 2) == [4, 4, 4, 4] * 2
    full = ["B 0 0", f"p 0 {8 * SMS} 0", "B 1 0", f"p 1 {8 * SMS} 0", "B 2 0", f"p 2 {8 * SMS} 0"]
    refill = ["e 0", "B 0 0", f"p 0 {8 * SMS} 0", "e 1", "B 1 0", f"p 1 {8 * SMS} 0", "e 2", "B 2 0", f"p 2 {8 * SMS} 0"]
    got = plan(full + refill * 3)
    for k in range(3, len(got) - 2, 3):
        assert sum(held(8 * SMS, lanes) for lanes in got[k:k + 3]) <= SMS


def test_a_resident_kernel_leaves_the_rest(plan):
    assert plan(["B 7 0", "h 7 136", "w 7", "b 0 0", "p 0 300 1", "e 0", "f 7", "b 0 0", "p 0 300 1", "b 0 0", "p 0 300 1"]) \
        == [1, 4, 4]
    # while it stays, callers that met once are not expected for ever
    three = ["b 0 0", "b 1 0", "b 2 0", "e 0", "e 1", "e 2"]
    assert plan(["B 7 0", "h 7 12", "w 7"] + three + ["b 0 0", "p 0 1000 1", "e 0"] * 3) == [1, 4, 4]


def test_nothing_stays_counted(plan):
    rng = random.Random(8)
    script = []
    state = ["off"] * 8
    for _ in range(3000):
        u = rng.randrange(1, 8)
        if state[u] == "off":
            script.append(rng.choice([f"b {u} 0", f"B {u} 0"]))
            state[u] = "on"
        elif state[u] == "on":
            script.append(rng.choice([f"p {u} {rng.randrange(1, 20000)} {rng.randrange(2)}", f"s {u} 5 1", f"h {u} 7", f"e {u}", f"w {u}"]))
            state[u] = {"e": "off", "w": "left"}.get(script[-1][0], "on")
        else:
            script.append(rng.choice([f"f {u}", f"e {u}", f"b {u} 0"]))
            state[u] = {"f": "left", "e": "off", "b": "on"}[script[-1][0]]
    script += [f"e {u}" for u in range(1, 8)]
    got = plan(script + ["b 0 0", "p 0 1 1", "e 0", "b 0 0", f"s 0 {SMS} 1", f"p 0 {8 * SMS} 1"])
    assert got[-3:] == [4, SMS, 4]
    assert all(v >= 1 for v in got)
    # another device's calls do not count
    assert plan(["b 1 1", "p 1 4736 1", "b 0 0", f"p 0 {8 * SMS} 1"]) == [1, 4]

"""What the branch and bound clears of its kept memo before a solve
(gtd_bnb_memo.h): every slot that could be taken for one of the solve's own,
and never more than the solve uses."""
import os
import random
import subprocess

import pytest

from gisbdw_gb300 import graphs as G

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "gtd_bnb_memo.h"
int main() {
  gtd::MemoSlots m;
  char op;
  unsigned long a, b;
  while (std::scanf(" %c %lu %lu", &op, &a, &b) == 3) {
    if (op == 'F') {
      m.fresh(a);
    } else {
      size_t first = 0;
      const size_t count = m.clear_before(a, b != 0, &first);
      std::printf("%zu %zu\n", first, count);
    }
  }
}
"""


@pytest.fixture(scope="module")
def clears(tmp_path_factory):
    d = tmp_path_factory.mktemp("memo")
    (d / "memo.cpp").write_text(PROGRAM)
    exe = str(d / "memo")
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "gisbdw_gb300", "csrc"), str(d / "memo.cpp"),
                    "-o", exe], check=True)

    def run(ops):
        text = "".join(f"{op} {a} {b}\n" for op, a, b in ops)
        out = subprocess.run([exe], input=text, check=True, capture_output=True, text=True).stdout.split()
        return [(int(out[i]), int(out[i + 1])) for i in range(0, len(out), 2)]
    return run


@pytest.mark.parametrize("seed", range(20))
def test_no_solve_meets_a_slot_it_could_take_for_its_own(clears, seed):
    rng = random.Random(seed)
    cap, ops = 0, []
    for _ in range(60):
        used = rng.choice([1, 2, 3, 5, 8, 13, 21, 40])
        if used > cap:
            cap = used
            ops.append(("F", cap, 0))
        ops.append(("S", used, int(rng.random() < 0.4)))
    got = iter(clears(ops))
    memo = []  # per slot: 'empty', 'plain' (without a number), or the number of a solve
    for number, (op, size, wide) in enumerate(ops):
        if op == "F":
            memo = ["plain"] * size  # whatever the memory held
            continue
        first, count = next(got)
        assert count <= size and (count == 0 or first + count <= size)
        for i in range(first, first + count):
            memo[i] = "empty"
        here = memo[:size]
        assert set(here) <= {"empty"} if wide else "plain" not in here, number
        memo[:size] = ["plain" if wide else number] * size


def test_repeated_solves_clear_what_they_use_or_nothing(clears):
    got = clears([("F", 64, 0), ("S", 64, 0), ("S", 64, 0), ("S", 1, 1), ("S", 1, 1), ("S", 1, 0), ("S", 64, 0)])
    assert [count for _, count in got] == [64, 0, 1, 1, 1, 0]


@pytest.mark.gpu
def test_one_wide_graph_after_a_large_batch_clears_its_own_slots_only():
    # 128 graphs leave a memo of 32 GiB: to clear all of it takes 4 ms at
    # 8 TB/s, one graph's 256 MiB 0.04 ms
    from gisbdw_gb300 import Handle
    h = Handle(0)
    h.bnb_solve_batch([G.path(5 + i % 8) for i in range(128)], deadline_ns=20 * 10**9)
    rest = []
    for _ in range(5):
        r = h.bnb_solve_batch([G.path(70)], deadline_ns=20 * 10**9)
        assert r["td"][0] == 7 and r["status"][0] == 0
        rest.append(r["stats"]["total_ms"] - r["stats"]["ms"])
    h.close()
    assert min(rest[1:]) < 2.5, rest  # the first one found the memo as a narrow solve leaves it

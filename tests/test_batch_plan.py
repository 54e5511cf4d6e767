"""The order of a batch's work (csrc/batch_plan.cpp, host only): tasks taken
in order, under the batch kernel's own rules of waiting, always go on, cover
every tile once, and never touch a slot before the circuit that held it is
done."""

import os
import subprocess
from collections import Counter, namedtuple

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
Wide = namedtuple("Wide", "index slot previous phases tiles")


@pytest.fixture(scope="module")
def planner(tmp_path_factory):
    from qevedo_simulator_b200 import build

    exe = str(tmp_path_factory.mktemp("plan") / "batch_plan")
    src = [os.path.join(ROOT, "tests", "batch_plan_main.cpp"), os.path.join(build.CSRC, "batch_plan.cpp")]
    subprocess.run([build.nvcc()] + build.host_compiler() + build.NVCC_FLAGS + src + ["-o", exe], check=True)

    def plan(circuits, tile, ctas, slots):
        text = f"{tile} {ctas} {slots}\n" + "".join(f"{n} {layers}\n" for n, layers in circuits)
        out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout
        wide, tasks = {}, []
        for line in out.splitlines():
            kind, *v = line.split()
            v = [int(x) for x in v]
            if kind == "wide":
                wide[v[0]] = Wide(*v[1:])
            else:
                tasks.append(tuple(v))
        return wide, tasks

    return plan


def before(x, phase):
    """Tiles of a circuit that are done before a phase begins (BatchWide::before)."""
    return 0 if phase == 0 else 1 + (phase - 1) * x.tiles


def may_run(task, wide, done):
    """Whether the kernel's waits let a task run."""
    circuit, phase = task[:2]
    x = wide[circuit]
    if phase == x.phases:
        return done[x.index] >= before(x, phase)
    if phase == 0 and x.previous >= 0:
        p = next(w for w in wide.values() if w.index == x.previous)
        return done[p.index] >= before(p, p.phases) + 1  # its results too
    return done[x.index] >= before(x, phase)


def wide_tasks(wide, tasks):
    return [t for t in tasks if t[0] in wide]


SPECS = [[(19, 2)] * 5, [(24, 1), (21, 0), (19, 4), (19, 1)], [(20, 0), (20, 0), (20, 0), (18, 2), (18, 2)],
         [(21, 2), (20, 0), (19, 5), (18, 0), (18, 0), (17, 1), (17, 0), (17, 9), (16, 1), (15, 3), (12, 4), (3, 0)]]


@pytest.mark.parametrize("circuits", SPECS)
@pytest.mark.parametrize("tile", [13, 14])
@pytest.mark.parametrize("slots", [1, 2, 3, 20])
def test_slots_are_taken_over_only_when_free(planner, circuits, tile, slots):
    wide, tasks = planner(circuits, tile, 16, slots)
    assert sorted(wide) == [i for i, (n, _) in enumerate(circuits) if n > tile]
    # In order, no task waits for a later one, and each pass takes each tile once.
    done, tiles = Counter(), Counter()
    for t in wide_tasks(wide, tasks):
        assert may_run(t, wide, done), t
        circuit, phase, first, count = t
        done[wide[circuit].index] += count
        for k in range(first, first + count):
            tiles[circuit, phase, k] += 1
    expected = {(i, 0, 0) for i in wide} | {(i, x.phases, 0) for i, x in wide.items()}
    expected |= {(i, p, k) for i, x in wide.items() for p in range(1, x.phases) for k in range(x.tiles)}
    assert set(tiles) == expected and set(tiles.values()) == {1}
    # A circuit whose results stay out holds its slot: whatever else runs, no
    # later circuit of the slot begins.
    holders = [(i, x) for i, x in sorted(wide.items(), key=lambda w: w[1].index) if x.phases]
    for i, x in holders:
        assert x.slot < slots
        later = {j for j, y in holders if y.slot == x.slot and y.index > x.index}
        done, left, ran = Counter(), wide_tasks(wide, tasks), True
        left.remove((i, x.phases, 0, 1))
        while ran:
            ran = False
            for t in list(left):
                if may_run(t, wide, done):
                    assert t[0] not in later, (t, i)
                    done[wide[t[0]].index] += t[3]
                    left.remove(t)
                    ran = True

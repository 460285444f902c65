"""Who ends a step (csrc/sfp_step.cuh: sfp_tail, sfp_last_block).  The last of
a launch's arriving blocks writes the next step's plan over what every block
of the launch reads when it starts, and blocks start whenever the GPU has
room for them.  So every block that has read the plan has to arrive, idle
ones too: then the last arrival follows every block's reads."""
import itertools
import os
import re

import pytest

import sfparticles_b200

SOURCE = open(os.path.join(os.path.dirname(sfparticles_b200.__file__), "csrc", "sfp_step.cuh")).read()
EVENT_BODIES = ("sfp_massive_body", "sfp_photon_body", "sfp_hot_body")


def body(name):
    """The text of a function, comments taken out."""
    at = SOURCE.index(f"void {name}(")
    at = SOURCE.index("{", SOURCE.index(")", at))
    depth, end = 0, at
    while True:
        depth += {"{": 1, "}": -1}.get(SOURCE[end], 0)
        end += 1
        if depth == 0:
            return re.sub(r"//[^\n]*", "", SOURCE[at:end])


def idle_blocks_arrive(name):
    """Whether every way out of the body, once it has read the plan, goes through sfp_tail."""
    text = body(name)
    text = text[text.index("sfp_view("):]
    outs = [m.start() for m in re.finditer(r"\breturn\b", text)]
    before = [re.split(r"[;{}]", text[:o].rstrip().rstrip(";"))[-1].strip() for o in outs]
    return all(s.startswith("sfp_tail(") for s in before) and text.rstrip().rstrip("}").rstrip().endswith("s_tab);")


def late_reads(grid, busy_now, busy_next, all_arrive):
    """Over every order in which the blocks of a launch start and arrive: whether some block starts after the step's
    end and finds work in the next plan."""
    arriving = grid if all_arrive else busy_now
    for order in itertools.permutations(range(grid)):
        plan, arrived = busy_now, 0
        for b in order:
            if plan != busy_now and b < plan:
                return True
            if all_arrive or b < plan:
                arrived += 1
                if arrived == arriving:
                    plan = busy_next
    return False


@pytest.mark.parametrize("name", EVENT_BODIES)
def test_no_block_reads_a_plan_that_its_launch_has_replaced(name):
    waited = re.search(r"sfp_last_block\(R->st, ([\w.]+)\)", body("sfp_tail")).group(1) == "gridDim.x"
    everyone = waited and idle_blocks_arrive(name)
    for grid, busy_now, busy_next in ((4, 1, 4), (5, 1, 2), (5, 3, 5), (5, 5, 5), (1, 1, 1)):
        assert not late_reads(grid, busy_now, busy_next, everyone), (grid, busy_now, busy_next)


def test_the_model_finds_the_fault():
    assert late_reads(4, 1, 4, False) and not late_reads(4, 4, 4, False)

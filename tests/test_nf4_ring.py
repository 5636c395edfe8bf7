"""The operand ring of the NF4 CTA-pair kernels (csrc/tc_gemm_nf4.cuh) under random schedules: parity barriers, loads that land in
any order, decode groups that skip phases, MMAs in order, two CTAs.  No k-block is decoded from another one's codes and no wait
is left over; without the wait for the stage's last k-block the model does find stale codes."""
import random
import re

import pytest

from .conftest import PKG_ROOT

SOURCE = (PKG_ROOT / "csrc" / "tc_gemm_nf4.cuh").read_text()
STAGES, GROUPS = (int(re.search(rf"NF4P_{n} = (\d+);", SOURCE).group(1)) for n in ("STAGES", "GROUPS"))


def passed(completions, parity):
    """mbarrier.try_wait.parity: the phase under way has the other parity."""
    return completions % 2 != parity


def simulate(blocks, stages, groups, wait_consumed, rng):
    ctas = [dict(empty=[0] * stages, codes_full=[0] * stages, codes=[-1] * stages, loading=[], issued=0,
                 block=list(range(groups)), waited=[False] * groups) for _ in range(2)]
    ready, arrived, issued, running = [0] * stages, [0] * stages, 0, []
    while issued < blocks or running:
        steps = [("commit",)] if running else []
        if issued < blocks and passed(ready[issued % stages], issued // stages % 2):
            steps.append(("mma",))
        for c in ctas:
            j = c["issued"]
            if j < blocks and passed(c["empty"][j % stages], (j // stages + 1) % 2):
                steps.append(("load", c))
            steps += [("land", c, j) for j in c["loading"]]
            for g, j in enumerate(c["block"]):
                if j >= blocks:
                    continue
                if not c["waited"][g]:
                    if not wait_consumed or j < stages or passed(c["empty"][j % stages], (j // stages + 1) % 2):
                        steps.append(("wait", c, g))
                elif passed(c["codes_full"][j % stages], j // stages % 2):
                    steps.append(("decode", c, g))
        if not steps:
            return "hang"
        what, *arg = rng.choice(steps) if rng.random() < 0.7 else rng.choice((steps[0], steps[-1]))
        if what == "commit":
            s = running.pop(0) % stages
            for c in ctas:
                c["empty"][s] += 1
        elif what == "mma":
            running.append(issued)
            issued += 1
        else:
            c = arg[0]
            if what == "load":
                c["loading"].append(c["issued"])
                c["issued"] += 1
            elif what == "land":
                c["loading"].remove(arg[1])
                c["codes_full"][arg[1] % stages] += 1
                c["codes"][arg[1] % stages] = arg[1]
            elif what == "wait":
                c["waited"][arg[1]] = True
            else:
                g, j = arg[1], c["block"][arg[1]]
                if c["codes"][j % stages] != j:
                    return "stale"
                c["block"][g] += groups
                c["waited"][g] = False
                arrived[j % stages] += 1
                if arrived[j % stages] == 2:
                    arrived[j % stages] = 0
                    ready[j % stages] += 1
    return "ok"


@pytest.mark.parametrize("wait_consumed,seen", [(True, {"ok"}), (False, {"ok", "stale"})])
def test_every_block_is_decoded_from_its_own_codes(wait_consumed, seen):
    rng = random.Random(0)
    assert {simulate(rng.randrange(1, 60), STAGES, GROUPS, wait_consumed, rng) for _ in range(500)} == seen

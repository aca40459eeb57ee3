"""Host rows of a launch: arrays filled from lists and from int32 arrays, against their definition row by row."""
import numpy as np
import pytest

from titanic_flash_41_b200.models.engine import StepPlan


@pytest.mark.parametrize("sizes", [(1,), (4, 4, 4), (3, 1, 200), (0, 5), ()])
@pytest.mark.parametrize("kind", [list, tuple, "int32", "int64"])
@pytest.mark.parametrize("logits", ["all", "last"])
def test_rows_of_a_plan(sizes, kind, logits):
    rng = np.random.default_rng(len(sizes))
    ids = [rng.integers(0, 129280, n) for n in sizes]
    give = lambda t: kind(t.tolist()) if callable(kind) else t.astype(kind)
    blocks = [(2 * i, 1000 * i + 7, give(t)) for i, t in enumerate(ids)]
    p = StepPlan.build(blocks, logits=logits)
    want = [[], [], [], [], [], []]
    for i, t in enumerate(ids):
        r0, n = len(want[0]), len(t)
        for j in range(n):
            for col, v in zip(want, (int(t[j]), 1000 * i + 7 + j, 2 * i, r0, 1000 * i + 7 + n - 1)):
                col.append(v)
        want[5] += list(range(r0, r0 + n)) if logits == "all" else [r0 + n - 1]
    got = (p.tokens, p.pos, p.region, p.first_row, p.last_pos, p.logit_rows)
    assert [g.tolist() for g in got] == want and all(g.dtype == np.int32 for g in got)
    assert p.group_rows == (sizes[0] if len(set(sizes)) == 1 else 1)
    assert [(r, s, [int(v) for v in t]) for r, s, t in p.blocks] == [(2 * i, 1000 * i + 7, t.tolist()) for i, t in enumerate(ids)]


def test_plan_refuses_what_does_not_fit_32_bits():
    StepPlan.build([(0, 2 ** 31 - 4, [1, 2, 3, 4])])
    for block in ((0, 2 ** 31 - 3, [1, 2, 3, 4]), (2 ** 31, 0, [1]), (0, 0, [2 ** 31])):
        with pytest.raises(OverflowError):
            StepPlan.build([block])
    with pytest.raises(TypeError):
        StepPlan.build([(0, 1.0, [1])])

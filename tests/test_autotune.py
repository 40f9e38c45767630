"""The autotuner's candidates and what it says of the one that it picks."""
from __future__ import annotations

import numpy as np
import pytest

from mojoalign_b200 import autotune as at


class Context:
    """Records the tunings set, in place of a GPU context."""

    def __init__(self):
        self.set = []

    def set_tuning(self, *tuning):
        self.set.append(tuning)

    def set_profiling(self, flags):
        pass


def test_every_candidate_runs_something_else():
    runs = set()
    for c in at.DEFAULT_CANDIDATES:
        full = tuple(c) + at.DEFAULTS[len(c):]
        # seed_kernels 2, 3 and 4 are the same passes
        runs.add((min(full[0], 2),) + full[1:])
    assert len(runs) == len(at.DEFAULT_CANDIDATES)


@pytest.mark.parametrize("best,fits", [((2, 1, 0, 1, 1, 1, 8, 4, 0, 1), True), ((2, 1, 0, 0), True),
                                       ((2, 2, 0, 1, 1, 1, 8, 4, 0, 1), False),
                                       ((2, 1, 0, 1, 1, 1, 8, 16, 0, 1), False), ((0, 1, 0, 1, 16, 32, 32), False)])
def test_the_result_tells_rounds_fitted_to_the_sample(best, fits):
    """Rounds fitted to the sample are not those of a call of another size."""
    candidates = [best, (2, 2, 0, 0, 1, 1, 9, 5, 0, 1), (1, 1, 0, 2, 1, 1, 32)]
    ctx = Context()

    def run():
        return {"pos": np.zeros(3)}, 1.0 if ctx.set[-1] == best else 2.0

    got = at.autotune(ctx, None, None, None, 3, False, 100, candidates=candidates, run=run)
    assert ctx.set[-1] == best and got.tuning == dict(zip(at.FIELDS, best + at.DEFAULTS[len(best):]))
    assert got.fitted is fits and [a["fitted"] for a in got.all_ms] == [fits, False, False]

"""The delay-rank tuner times every rank that acts differently once: a rank above
the 16 sites of an update window acts as 16."""
import pytest

from dqmc_b200 import batch


class _Chain:
    def __init__(self, n):
        self.N = n


@pytest.mark.parametrize("n,candidates,timed", [
    (64, (4, 8, 16, 32), [4, 8, 16]), (64, (32, 16, 4), [32, 4]), (9, (4, 8, 16), [4, 8]), (64, (64, 32), [64])])
def test_ranks_that_act_alike_are_timed_once(monkeypatch, n, candidates, timed):
    got = []
    monkeypatch.setattr(batch, "time_sweep", lambda sims, kd, device: got.append(kd) or 1.0 / len(got))
    assert batch.autotune_delay([_Chain(n)], candidates) == timed[-1]
    assert got == timed

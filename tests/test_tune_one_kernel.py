"""The ensemble autotuner leaves the knobs alone that shape nothing where the substeps run in one
cooperative kernel: no trial, no choice."""
from brownian_gb300 import ENS_AUX, ENS_EVENTS, tune


class FakeEnsemble:
    one_kernel = True

    def __init__(self):
        self.tried = {}

    def set_launch(self, which, per_system=1, block=32):
        self.tried.setdefault(which, set()).add((per_system, block))

    def step(self, n=1):
        pass


def test_knobs_without_effect_are_not_tuned():
    ens = FakeEnsemble()
    res = tune.autotune(ens, steps=1)
    for which, name in ((ENS_EVENTS, "events_blocks_per_system"), (ENS_AUX, "aux_threads_per_colloid")):
        assert ens.tried[which] == {tune.DEFAULTS[name]}
        assert res["choice"][name] == list(tune.DEFAULTS[name])
    assert {t["knob"] for t in res["log"] if "knob" in t} == set(tune.CANDIDATES) - set(tune.PER_STAGE_ONLY)

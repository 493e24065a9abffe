"""What the autotuner times and sets, with the library and the clock replaced: a knob that the timed kernels do not
read keeps its value, and each plume kernel is timed as often as the other."""
import pytest

from bug_defense_b200 import _lib, campaign


class _Engine:
    laser_power = 1.0

    def step_epochs(self, n):
        pass


@pytest.fixture
def fake(monkeypatch):
    knobs = {_lib.TUNE_MC_BLOCKS_PER_SM: 0, _lib.TUNE_STENCIL_XC: 8, _lib.TUNE_PLUME_XC: 5,
             _lib.TUNE_PLUME_KERNEL: _lib.PLUME_KERNEL_DIRECT, _lib.TUNE_STENCIL_CAP: 0}
    sets, timed = [], []

    def call(name, knob, value):
        if name == "bd_tune_set":
            knobs[knob] = value
            sets.append((knob, value))
        else:
            assert name == "bd_tune_get"
            value._obj.value = knobs[knob]

    def epoch_ms(eng, n, laser):
        timed.append((dict(knobs), laser))
        return 1.0 + 0.1 * (knobs[_lib.TUNE_PLUME_KERNEL] == _lib.PLUME_KERNEL_COMPACT) - 0.001 * len(timed)

    monkeypatch.setattr(_lib, "call", call)
    monkeypatch.setattr(campaign, "_epoch_ms", epoch_ms)
    monkeypatch.setattr(campaign, "_stage_ms", lambda *a, **k: None)
    return knobs, sets, timed


def test_plume_planes_keep_their_value(fake):
    knobs, sets, timed = fake
    out = campaign.autotune(_Engine)
    assert knobs[_lib.TUNE_PLUME_XC] == out["plume_xc"] == 5
    assert all(knob != _lib.TUNE_PLUME_XC for knob, _ in sets)
    assert [(k, x) for k, x, _ in out["trials"]["plume"]] == [(_lib.PLUME_KERNEL_DIRECT, None),
                                                            (_lib.PLUME_KERNEL_COMPACT, None)]
    # the plume trials follow the two substep knobs' and come before the photons'
    n0 = len(out["trials"]["stencil_xc"]) + len(out["trials"]["stencil_cap"])
    plume = [k[_lib.TUNE_PLUME_KERNEL] for k, laser in timed[n0:] if not laser]
    assert plume.count(_lib.PLUME_KERNEL_DIRECT) == plume.count(_lib.PLUME_KERNEL_COMPACT) == 2
    assert out["plume_kernel"] == _lib.PLUME_KERNEL_DIRECT


def test_named_plume_planes_are_searched(fake):
    knobs, _, _ = fake
    out = campaign.autotune(_Engine, candidates={_lib.TUNE_PLUME_XC: [2, 4]})
    assert [(k, x) for k, x, _ in out["trials"]["plume"]] == [(4, 2), (4, 4), (6, None)]
    assert out["plume_xc"] == knobs[_lib.TUNE_PLUME_XC] in (2, 4)

"""The hand-off protocol of the one-vector matvec (yule_b200/csrc/qmv_digits.cu) on a model under random interleavings: with
copies that arrive, and with copies that stop arriving.  The variants that go wrong then (a warp that gave up does not wait for
the others; as many barriers as buffers; it releases its stages) must be caught, so that a green run means something."""

import pytest

from qmv_digits_model import Config, ProtocolViolation, finish_buffers, run

# (ring slots, stages per unit, warps): short rows with a deep ring, longer rows, a pair's two matrices; and half the warps
RINGS = [(1, 1, 16), (4, 1, 16), (6, 1, 16), (5, 2, 16), (3, 7, 16), (4, 1, 8), (2, 3, 8)]


def failures(cfg: Config, seeds) -> list:
    bad = []
    for seed in seeds:
        try:
            run(cfg, seed)
        except ProtocolViolation as e:
            bad.append((seed, str(e)))
    return bad


@pytest.mark.parametrize("slots,stages,warps", RINGS)
def test_sums_are_complete_and_kept(slots, stages, warps):
    cfg = Config(warps=warps, slots=slots, stages_per_unit=stages, finish=finish_buffers(slots, stages), units=14)
    assert failures(cfg, range(40)) == []


@pytest.mark.parametrize("slots,stages,warps", RINGS)
def test_everybody_leaves_when_copies_stop(slots, stages, warps):
    for fail_at in (0, 40, 150, 400):
        cfg = Config(warps=warps, slots=slots, stages_per_unit=stages, finish=finish_buffers(slots, stages), units=14, fail_at=fail_at)
        assert failures(cfg, range(15)) == []


def test_model_catches_warps_that_run_ahead_and_too_few_buffers():
    ahead = Config(slots=2, finish=3, units=12, dead_waits=False)
    assert failures(ahead, range(10)) == []  # sound as long as every copy arrives
    ahead.fail_at = 150
    assert any("deadlock" in why for _, why in failures(ahead, range(60)))
    as_many = Config(slots=4, finish=5, units=14, fail_at=150, more_barriers=0)
    assert any("deadlock" in why for _, why in failures(as_many, range(60)))
    again = Config(slots=2, finish=3, units=12, fail_at=150, dead_keeps=False)
    assert any("arrival beyond" in why for _, why in failures(again, range(60)))
    assert failures(Config(slots=6, finish=2, units=14), range(40))

"""The hand-off protocol of the tcgen05 GEMM kernel (yule_b200/csrc/qgemm_tc.cu) checked on a model under random
interleavings: the ring sizes the kernel is built with, a sweep around them, waits that run out, and variants that are known to be
broken, which the model must catch (so that a green run means something)."""

import os
import re

import pytest

from gemm_pipeline_model import Config, ProtocolViolation, run

with open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yule_b200", "csrc", "qgemm_tc.cu")) as f:
    SOURCE = f.read()


def kernel_rings() -> dict:
    """Ring sizes of every instantiation, from the expressions in the source: C++ that is Python once its names are given."""
    def constant(name):
        return int(re.search(rf"\b{name} = (\d+)[,;]", SOURCE).group(1))

    def expression(text, **names):
        text = re.sub(r"(\d)u\b", r"\1", text).replace("&&", " and ").replace("!", " not ").replace("/", "//")
        pick = re.fullmatch(r"(.*?)\?(.*?):(.*)", text)
        if pick:
            text = f"({pick[2]}) if ({pick[1]}) else ({pick[3]})"
        return eval(text, {}, names)  # noqa: S307 (our own source)

    def tile(name, **names):
        return expression(re.search(rf"static constexpr \w+ {name} = (.*?);", SOURCE).group(1).replace("(GENERIC ? 2 : 1)", "GROUPS"), **names)

    rings = {}
    for generic in (False, True):
        for bn in (32, 64, 128):
            names = {"BN": bn, "GENERIC": generic, "GROUPS": 2 if generic else 1, "kBK": constant("kBK"), "kStages": constant("kStages")}
            names["KG"] = expression(re.search(r"groups_per_stage\(uint32_t bn, bool generic\) \{\s*return (.*?);", SOURCE).group(1), bn=bn, generic=generic)
            for name in ("MERGED", "SPB", "kACols", "kMainCols", "NBUF"):
                names[name] = tile(name, **names)
            raw = expression(re.search(r"raw_slots_for\(uint32_t bn\) \{ return (.*?);", SOURCE).group(1), bn=bn, kRawSlots=constant("kRawSlots"))
            rings[f"{'other' if generic else 'q4k'}-{bn}"] = Config(stages=names["kStages"], nbuf=names["NBUF"], raw_slots=raw, stages_per_unit=names["SPB"],
                                                                    units=9, min_term=not generic)
    return rings


RINGS = kernel_rings()


def failures(cfg: Config, seeds) -> list:
    bad = []
    for seed in seeds:
        try:
            run(cfg, seed)
        except ProtocolViolation as e:
            bad.append((seed, str(e)))
    return bad


def test_the_ring_sizes_in_the_source():
    """So that a change of the source that these tests do not follow is seen."""
    assert {k: (c.stages, c.nbuf, c.raw_slots, c.stages_per_unit) for k, c in RINGS.items()} == {
        "q4k-32": (4, 4, 6, 2), "q4k-64": (4, 3, 6, 4), "q4k-128": (4, 3, 3, 4), "other-32": (4, 4, 6, 4), "other-64": (4, 2, 6, 4), "other-128": (4, 2, 3, 4)}


@pytest.mark.parametrize("name", list(RINGS))
def test_protocol_holds_at_the_kernel_ring_sizes(name):
    assert failures(RINGS[name], range(120)) == []


def test_protocol_holds_around_them():
    for stages in (2, 4, 6):
        for raw in (2, 4):
            for nbuf, min_term in ((3, True), (5, True), (2, False), (3, False)):
                cfg = Config(stages=stages, nbuf=nbuf, raw_slots=raw, stages_per_unit=2, units=6, min_term=min_term)
                assert failures(cfg, range(12)) == [], cfg


def test_full_size_warp_counts():
    assert failures(Config(producer_warps=8, drain_warps=8, units=5), range(30)) == []


@pytest.mark.parametrize("name", list(RINGS))
def test_everybody_gets_to_the_end_when_waits_run_out(name):
    for fail_at in (0, 40, 150, 400):
        cfg = RINGS[name]
        assert failures(Config(**{**vars(cfg), "fail_at": fail_at}), range(40)) == []


def test_an_unpacking_warp_that_leaves_the_barriers_is_caught():
    bad = [f for at in range(20, 400, 20) for f in failures(Config(**{**vars(RINGS["other-128"]), "fail_at": at, "producers_leave": True}), range(20))]
    assert any("deadlock" in msg for _, msg in bad), "the model no longer finds the hang"


def test_an_accumulator_ring_that_is_too_short_is_caught():
    """With one accumulator fewer than the parities need, a warp takes the phase before last for the last."""
    assert failures(Config(**{**vars(RINGS["q4k-128"]), "nbuf": 2}), range(200)), "the model no longer finds it"


def test_teams_on_alternate_stages_are_caught():
    """Two teams of unpacking warps on alternate stages wait on every other phase of a stage's `empty` barrier; a
    parity wait cannot tell phase k from phase k - 2, so with an odd ring a team that is ahead passes its wait early and
    overwrites what has not been read."""
    bad = failures(Config(teams=True, stages=3), range(60))
    assert bad, "the model no longer finds the overwrite"

"""Every entry point that takes a context ends the chain of dependent launches or goes on with it: one that did neither would leave its outputs out of the list by
which a matvec knows what it must not read before it waits.  From the sources, on the CPU (the mistake is a race on memory)."""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yule_b200", "csrc")
# what enqueues nothing, or waits for the stream behind what it enqueues
NEITHER = {f"yule_cuda_{n}" for n in ("destroy", "launch_count", "tp_init", "selftest_bounded_wait", "runner_buffer", "runner_destroy", "runner_position", "runner_reset",
                                     "runner_reset_batch", "runner_set_tensor")}


def entry_points():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            text = f.read()
        for m in re.finditer(r"^(?:extern \"C\" |static )?int32_t (\w+)\((?:yule_cuda_ctx \*ctx|yule_cuda_runner \*r)\b[^)]*\) \{\n(.*?)^\}", text, re.M | re.S):
            if m[1].startswith("yule_cuda_") or m[1] in ("qmv_common", "finalize"):
                yield m[1], m[2]


BODIES = dict(entry_points())


def ends(body):
    if re.search(r"CTX_(GUARD|ENQUEUE)\(ctx\)|ctx->take_chain\(\)", body):
        return True
    called = set(re.findall(r"\b(\w+)\((?:ctx|r)\b", body)) & set(BODIES)
    return any(ends(BODIES[c]) for c in called)


@pytest.mark.parametrize("name", sorted(BODIES))
def test_the_chain_ends_or_goes_on(name):
    assert name in NEITHER or ends(BODIES[name])


def test_the_entry_points_are_found():
    assert len(BODIES) > 40 and {"yule_cuda_multihead_attention_static", "yule_cuda_rms_norm", "qmv_common", "yule_cuda_runner_prefill"} <= set(BODIES)

"""The sampler where one CTA finishes it over the candidates that the top-k descent leaves (finish_few in csrc/sampler.cu), against the oracle: the limits of that
path, and equal probabilities at the top-k threshold and where the mass reaches top_p, spread over all CTAs of the cluster."""

import numpy as np
import pytest

from test_gpu_sampler import near_boundary
from yule_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("top_k", [1, 31, 40, 254, 255, 256, 300])
@pytest.mark.parametrize("n", [3, 9, 260, 5000, 32003])
def test_limits(backend, oracle, n, top_k):
    logits = (4.0 * synth.normal(50 + n, n)).astype(np.float32)
    lh = backend.upload(logits)
    for kw in (dict(temperature=0.8, top_p=0.9, top_k=top_k, repetition_penalty=1.0, min_p=0.0),
               dict(temperature=1.5, top_p=1.0, top_k=top_k, repetition_penalty=1.0, min_p=0.02),
               dict(temperature=1.0, top_p=0.0, top_k=top_k, repetition_penalty=1.0, min_p=1.0)):
        for r in (0.0, 0.05, 0.31, 0.77, 0.98):
            if r == 0.0 or not near_boundary(oracle, logits, r, kw, np.zeros(0, np.uint32)):
                assert backend.sample(lh, n, r, **kw) == oracle.sample(logits, r, **kw)
    backend.free(lh)


@pytest.mark.parametrize("levels,n", [((5, 30, 300), 4000), ((1, 2, 250), 4000), ((20, 200, 1000), 4000), ((300, 10, 10), 4000), ((2, 300, 9), 4000)])
def test_ties(backend, oracle, levels, n):
    """So many tokens of the largest, the second and the third value, dealt over the vocabulary; the others lie far below."""
    logits = np.full(n, -20.0, np.float32)
    at = np.random.default_rng(sum(levels)).permutation(n)
    for i, m in enumerate(levels):
        logits[at[:m]], at = 5.0 - 1.5 * i, at[m:]
    lh = backend.upload(logits)
    for top_k in (1, 4, 39, 240):
        for top_p in (0.2, 0.5, 0.93, 1.0):
            kw = dict(temperature=1.0, top_p=top_p, top_k=top_k, repetition_penalty=1.0, min_p=0.0)
            for r in (0.013, 0.37, 0.61, 0.94):
                got, want = backend.sample(lh, n, r, **kw), oracle.sample(logits, r, **kw)
                # Which of equal tokens stay at the boundary is the reference's to choose: the same value is asked for, and with all of them the same token.
                assert logits[got] == logits[want] or near_boundary(oracle, logits, r, kw, np.zeros(0, np.uint32))
                if top_p == 1.0 and not near_boundary(oracle, logits, r, kw, np.zeros(0, np.uint32)):
                    assert got == want
    backend.free(lh)


def test_not_finite(backend):
    for bad in (np.nan, np.inf, -np.inf):
        logits = synth.normal(3, 1000).astype(np.float32)
        logits[::3] = bad
        lh = backend.upload(logits)
        assert 0 <= backend.sample(lh, 1000, 0.4) < 1000
        backend.free(lh)

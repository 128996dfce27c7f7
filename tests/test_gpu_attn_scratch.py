"""The scratch of the attention entry point (csrc/api.cu), shared by its two routes: clusters for short contexts, splits for long ones.  The lengths
lie on both sides of the line, in both orders; the group of four query heads is one where the routes want different numbers of tickets."""

import numpy as np
import pytest
import torch

from test_gpu_attn_cluster import TOL, attention64
from yule_b200 import CudaB200Backend, synth

pytestmark = pytest.mark.gpu
HEADS, KV, HD = 32, 8, 128
STRIDE = KV * HD


@pytest.fixture
def host():
    class Host:
        def __init__(self, longest):
            self.b = CudaB200Backend(0)
            self.data = synth.normal(1, HEADS * HD), synth.normal(2, longest * STRIDE), synth.normal(3, longest * STRIDE)
            self.q, self.k, self.v = (self.b.upload(a) for a in self.data)
            self.out = self.b.allocate(HEADS * HD * 4)

        def call(self, seq):
            self.b.multihead_attention(self.q, self.k, self.v, self.out, HD, seq, HEADS, KV, STRIDE)

        def right(self, seq):
            q, K, V = self.data
            ref = attention64(q, K.reshape(-1, STRIDE)[:seq], V.reshape(-1, STRIDE)[:seq], HEADS, KV, HD)
            return np.abs(self.b.download(self.out, HEADS * HD) - ref).max() <= TOL * np.abs(ref).max()

    made = []

    def make(longest):
        made.append(Host(longest))
        return made[-1]

    yield make
    for h in made:
        h.b.close()


@pytest.mark.parametrize("one,other", [(4000, 1000), (1000, 4000), (2000, 3000)])
def test_turns_between_long_and_short_allocate_once(host, one, other):
    h = host(4000)
    for seq in (one, other):
        h.call(seq)
    h.b.synchronize()
    free = torch.cuda.mem_get_info(0)[0]
    for _ in range(200):
        for seq in (one, other):
            h.call(seq)
    h.b.synchronize()
    assert torch.cuda.mem_get_info(0)[0] == free
    for seq in (one, other, one):
        h.call(seq)
        assert h.right(seq)


@pytest.mark.parametrize("before,captured", [((4000,), 1000), ((2000,), 4000), ((1000, 4000), 1000), ((4000, 1000), 4000), ((300, 2000), 4000)])
def test_a_call_that_the_scratch_is_large_enough_for_can_be_captured(host, before, captured):
    h = host(4000)
    for seq in before:
        h.call(seq)
    h.b.graph_begin()
    h.call(captured)
    graph = h.b.graph_end()
    for seq in (1000, 4000):  # what runs between the capture and the replay
        h.call(seq)
    for _ in range(2):
        h.b.graph_launch(graph)
        assert h.right(captured)

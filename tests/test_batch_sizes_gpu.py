"""Batches on both sides of the lines at which the counting and packing warps
take their items from the start, one by one, ahead, and several at a time: from
a few slice components to 150,000 (4,736 warps are resident)."""

import numpy as np
import pytest

import rivet_prores_b200 as P
from oracle import oracle as O
from tests.util import to_config, to_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,targets", [
    (32, 16, [400]),
    (1248, 640, [200000]),           # 9,360 components: two a warp
    (1920, 1088, [250000, 500000]),  # 48,960: ten a warp, taken ahead
    (1920, 1088, [40000, 250000, 500000, 1000000, 2500000, 1 << 30]),  # 146,880: three at a time
])
def test_every_frame_of_the_batch_is_the_oracles(width, height, targets):
    rng = np.random.Generator(np.random.PCG64(width))
    pic = O.test_frame(width, height, 2, 10, 4, 1)
    pic.data[:] = np.clip(pic.data + rng.normal(0, 60, pic.data.size), 4, 1019).astype(pic.data.dtype)
    cfgs = [O.Config(3, log2_slice_mbs=0, target_frame_bytes=t) for t in targets]
    got = P.Encoder(to_config(cfgs[0])).encode_batch([to_frame(pic)] * len(cfgs), [to_config(c) for c in cfgs])
    for cfg, g in zip(cfgs, got):
        k, msg, want = O.encode(cfg, pic)
        assert k == O.OK, msg
        assert not isinstance(g, P.Error) and g == want, cfg.target_frame_bytes

"""The rate control's passes of one to three probes against the oracle: targets
from below the coarsest quantiser's size up to the finest's, so that the
bisection ends at either bound and on both sides of 112 and 56. One batch of
few slices, whose later passes take three probes, and one of many slices,
whose passes take one."""

import numpy as np
import pytest

import rivet_prores_b200 as P
from oracle import oracle as O
from tests.util import to_config, to_frame

pytestmark = pytest.mark.gpu


def _cases(width, height, log2, targets, profile, interlace):
    rng = np.random.Generator(np.random.PCG64(width + profile))
    pic = O.test_frame(width, height, 3 if profile >= 4 else 2, 10, 4, 1)
    pic.interlace = interlace
    pic.data[:] = np.clip(pic.data + rng.normal(0, 60, pic.data.size), 4, 1019).astype(pic.data.dtype)
    return [(O.Config(profile, log2_slice_mbs=log2, target_frame_bytes=int(t)), pic)
            for t in targets]


def _check(cases):
    got = P.Encoder(to_config(cases[0][0])).encode_batch([to_frame(p) for _, p in cases],
                                                        [to_config(c) for c, _ in cases])
    for (cfg, pic), g in zip(cases, got):
        k, msg, want = O.encode(cfg, pic)
        assert k == O.OK, msg
        assert not isinstance(g, P.Error) and g == want, cfg.target_frame_bytes


@pytest.mark.parametrize("profile,interlace", [(3, 0), (4, 1)])
def test_few_slices(profile, interlace):
    _check(_cases(176, 64, 1, np.geomspace(300, 60000, 24), profile, interlace))


def test_many_slices():
    _check(_cases(1920, 1088, 0, (40000, 250000, 500000, 1000000, 2500000, 1 << 30), 3, 0))

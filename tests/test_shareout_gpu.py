"""The share-out against the oracle: fewer slices than a warp settles at once,
one more, and several times as many; targets that leave a uniform quantiser
from 224 down to 1; and pictures whose slices step by none, by the window, by
the deep ladder and past it (flat slices reach quantiser 1 from any other, so
from above 133 they need levels that only the share-out costs)."""

import numpy as np
import pytest

import rivet_prores_b200 as P
from oracle import oracle as O
from tests.util import to_config, to_frame

pytestmark = pytest.mark.gpu


def _picture(kind, width, height, chroma, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    pic = O.test_frame(width, height, chroma, 10, 4, seed)
    noise = rng.normal(0, 150, pic.data.size)
    if kind == "half":  # the left half of the luma rows
        noise[np.arange(noise.size) % width < width // 2] = 0
        pic.data[:] = 512
    elif kind == "few":  # a few strong samples in a flat field
        noise[rng.random(noise.size) < 0.995] = 0
        pic.data[:] = 512
    pic.data[:] = np.clip(pic.data + noise, 4, 1019).astype(pic.data.dtype)
    return pic


@pytest.mark.parametrize("kind", ["noise", "half", "few"])
@pytest.mark.parametrize("width,height,log2", [(64, 32, 3), (176, 64, 0), (528, 16, 0), (496, 64, 0), (720, 80, 1)])
def test_steps_are_the_oracles(kind, width, height, log2):
    cases = []
    for profile, chroma in ((3, 2), (4, 3)):
        pic = _picture(kind, width, height, chroma, width + profile)
        least = len(O.encode(O.Config(profile, log2_slice_mbs=log2, target_frame_bytes=1), pic)[2])
        most = len(O.encode(O.Config(profile, log2_slice_mbs=log2, target_frame_bytes=1 << 30), pic)[2])
        for target in np.geomspace(least, most + 16, 9):
            cases.append((O.Config(profile, log2_slice_mbs=log2, target_frame_bytes=int(target)), pic))
    got = P.Encoder(to_config(cases[0][0])).encode_batch([to_frame(p) for _, p in cases],
                                                        [to_config(c) for c, _ in cases])
    for (cfg, pic), g in zip(cases, got):
        k, msg, want = O.encode(cfg, pic)
        assert k == O.OK, msg
        assert not isinstance(g, P.Error) and g == want, (cfg.profile, cfg.target_frame_bytes)

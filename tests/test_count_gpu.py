"""The warp-wide bit count of the rate control against the oracle, at the
edges of its ways through a component: few live chunks (their list), most
chunks live (all in turn), run and level symbols past its tables, and levels
too large for its half-word entries. 176 columns make slices of 8, 2 and 1
macroblocks, so components of 2 to 32 blocks."""

import numpy as np
import pytest

import rivet_prores_b200 as P
from oracle import oracle as O
from tests.util import to_config, to_frame

pytestmark = pytest.mark.gpu


def _picture(kind, chroma, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    depth = 8 if kind.startswith("out") else 10
    p = O.test_frame(176, 64, chroma, depth, 4, seed)
    n = p.data.size
    if kind == "noise":
        p.data[:] = rng.integers(64, 940, n)
    elif kind == "faint":  # a flat field with a few single-sample marks: sparse, long runs
        p.data[:] = 512
        p.data[rng.integers(0, n, n // 300)] = 600
    elif kind == "strong":  # two-valued rows: large levels beside zeros
        p.data[:] = np.where(rng.random(n) < 0.5, 4, 1019)
    else:  # samples past the depth's range, which the codec takes as they are
        p.data[:] = np.where(rng.random(n) < 0.5, 0, {"out2000": 2000, "out8191": 8191, "out65535": 65535}[kind])
    return p


@pytest.mark.parametrize("kind", ["noise", "faint", "strong", "out2000", "out8191", "out65535"])
def test_every_way_of_counting_gives_the_oracles_packet(kind):
    cases = []
    for chroma, profile in ((2, 3), (3, 4)):
        for log2 in range(4):
            for target in (None, 1 << 30, 6000):
                cases.append((O.Config(profile, log2_slice_mbs=log2, target_frame_bytes=target),
                              _picture(kind, chroma, 100 * profile + log2)))
    got = P.Encoder(to_config(cases[0][0])).encode_batch([to_frame(p) for _, p in cases],
                                                        [to_config(c) for c, _ in cases])
    for i, ((cfg, pic), g) in enumerate(zip(cases, got)):
        k, msg, want = O.encode(cfg, pic)
        assert k == O.OK, msg
        assert not isinstance(g, P.Error) and g == want, (kind, i)


@pytest.mark.parametrize("weights", ["least", "most", "mixed"])
def test_quantiser_tables_of_extreme_weights(weights):
    """The tables the device builds, over coarse and fine quantisers, both
    scans and both matrices, sets of different frames side by side."""
    cases = []
    for i, (chroma, profile) in enumerate(((2, 3), (3, 4), (2, 1))):
        rng = np.random.Generator(np.random.PCG64(i))
        luma, chroma_w = ((bytes([2] * 64), bytes([63] * 64)) if weights == "least" else
                          (bytes([63] * 64), bytes([2] * 64)) if weights == "most" else
                          (bytes(int(v) for v in rng.integers(2, 64, 64)), None))
        for interlace in range(2):
            for target in (None, 1 << 30, 4000):
                p = _picture("noise" if target else "strong", chroma, 7 * i + interlace)
                p.interlace = interlace
                cases.append((O.Config(profile, log2_slice_mbs=i, luma_matrix=luma, chroma_matrix=chroma_w,
                                       target_frame_bytes=target), p))
    got = P.Encoder(to_config(cases[0][0])).encode_batch([to_frame(p) for _, p in cases],
                                                        [to_config(c) for c, _ in cases])
    for i, ((cfg, pic), g) in enumerate(zip(cases, got)):
        k, msg, want = O.encode(cfg, pic)
        assert k == O.OK, msg
        assert not isinstance(g, P.Error) and g == want, (weights, i)

"""The warp-synchronous entropy decoder against the oracle where its steps
part ways: components whose levels pass the prefix tables, packets with
nothing but escapes or nothing at all, warps of components of very different
lengths, alpha of long runs, of a code a sample and of both, in slices and
planes whose rows do not fill its 8-sample groups, and data cut anywhere."""

import numpy as np
import pytest

import rivet_prores_b200 as P
from oracle import oracle as O
from tests.util import assert_decode_matches

pytestmark = pytest.mark.gpu


def _alpha(kind, w, h, rng):
    a = np.full((h, w), 65535, np.uint16)
    if kind == "noise":
        a[:] = rng.integers(0, 65536, (h, w))
    elif kind == "steps":  # small differences (the short codes) and runs of 1 to 40
        a[:] = np.repeat(rng.integers(0, 60, h * w), rng.integers(1, 41, h * w))[:h * w].reshape(h, w)
    elif kind == "mixed":
        a[:, w // 2:] = rng.integers(0, 65536, (h, w - w // 2))
    return a.ravel()


@pytest.mark.parametrize("bits", [1, 2])
@pytest.mark.parametrize("kind", ["flat", "noise", "steps", "mixed"])
def test_alpha_runs_and_rows(bits, kind):
    packets = []
    for i, (w, h) in enumerate([(16, 16), (33, 20), (121, 35), (200, 48), (7, 5)]):
        p = O.test_frame(w, h, 3, 16, 6, i)
        p.interlace = i % 3
        p.alpha = _alpha(kind, w, h, np.random.Generator(np.random.PCG64(i)))
        k, msg, packet = O.encode(O.Config(4, log2_slice_mbs=i % 4, alpha=bits), p)
        assert k == O.OK, msg
        packets.append(packet)
    for depth in (8, 12, 16):
        for i, (g, packet) in enumerate(zip(P.Decoder.with_bit_depth(depth).decode_batch(packets), packets)):
            assert_decode_matches(g, O.decode(packet, depth), f"{kind} {i} at {depth} bits")


@pytest.mark.parametrize("kind", ["levels", "uneven", "cut"])
def test_components_of_every_length(kind):
    packets = []
    for i in range(6):
        rng = np.random.Generator(np.random.PCG64(50 + i))
        p = O.test_frame(400, 64, 2 if i % 2 else 3, 12, 12, i)
        if kind == "levels":
            p.data[:] = rng.integers(0, 4096, p.data.size)
        else:  # detail in a few slices only
            p.data[:] = 2000
            for _ in range(4):
                at = int(rng.integers(0, p.data.size - 3000))
                p.data[at:at + 3000] = rng.integers(0, 4096, 3000)
        k, msg, packet = O.encode(O.Config(3 if i % 2 else 5, log2_slice_mbs=i % 4, target_frame_bytes=1 << 30), p)
        assert k == O.OK, msg
        if kind == "cut":
            packet = bytearray(packet)
            for at in rng.integers(200, len(packet), 3):
                packet[at:at + 6] = bytes(6) if at % 2 else b"\xff" * 6
            packet = bytes(packet)
        packets.append(packet)
    for i, (g, packet) in enumerate(zip(P.Decoder.new().decode_batch(packets), packets)):
        assert_decode_matches(g, O.decode(packet), f"{kind} {i}")

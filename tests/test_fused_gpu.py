"""The fused decoder (decode_fused, off by default) against the oracle: planes,
alpha and error messages, with coefficients held in one byte and in two, from
one slice a block to the most its shared memory takes. Its readers, its slots
and its transform are not the two-kernel decoder's."""

import numpy as np
import pytest

import rivet_prores_b200 as P
from oracle import oracle as O
from tests.test_entropy_gpu import _alpha
from tests.util import assert_decode_matches

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[(b, n) for b in (1, 2) for n in (512, 6144, 65536)], ids=lambda p: f"{p[0]}B-{p[1]}")
def fused(request):
    ctx = P.context(0)
    saved = ctx.tuning
    ctx.set_tuning(P.Tuning(decode_fused=1, decode_slot_bytes=request.param[0], decode_slot_positions=request.param[1]))
    yield
    ctx.set_tuning(saved)


def _encode(p, profile, **kw):
    k, msg, packet = O.encode(O.Config(profile, **kw), p)
    assert k == O.OK, msg
    return packet


def _packets(kind):
    out = []
    for i in range(6):
        rng = np.random.Generator(np.random.PCG64(50 + i))
        chroma = 2 if i % 2 else 3
        if kind in ("flat", "noise", "steps", "mixed"):  # alpha
            w, h = [(16, 16), (33, 20), (121, 35), (200, 48), (7, 5), (64, 64)][i]
            p = O.test_frame(w, h, 3, 16, 6, i)
            p.interlace = i % 3
            p.alpha = _alpha(kind, w, h, rng)
            out += [_encode(p, 4, log2_slice_mbs=i % 4, alpha=bits) for bits in (1, 2)]
            continue
        w, h = [(400, 64), (240, 33), (119, 17), (16, 16), (41, 64), (233, 50)][i]
        p = O.test_frame(w, h, chroma, 12, 12, i)
        p.interlace = i % 3
        if kind == "levels":  # codes past the tables, values past the slots
            p.data[:] = rng.integers(0, 4096, p.data.size)
        elif kind == "uneven":
            p.data[:] = 2000
            at = int(rng.integers(0, p.data.size // 2))
            p.data[at:at + 300] = rng.integers(0, 4096, p.data[at:at + 300].size)
        packet = _encode(p, 3 if i % 2 else 5, log2_slice_mbs=i % 4,
                         target_frame_bytes=None if kind == "picture" else 1 << 30)
        if kind == "cut":
            packet = bytearray(packet)
            for at in rng.integers(170, len(packet), 3):
                packet[at:at + 6] = bytes(6) if at % 2 else b"\xff" * 6
            packet = bytes(packet)
        out.append(packet)
    return out


@pytest.mark.parametrize("kind", ["picture", "levels", "uneven", "cut", "flat", "noise", "steps", "mixed"])
def test_the_fused_decoder_gives_the_oracles_pictures(fused, kind):
    packets = _packets(kind)
    for depth in (None, 16):
        got = P.Decoder(depth).decode_batch(packets)
        for i, (g, packet) in enumerate(zip(got, packets)):
            assert_decode_matches(g, O.decode(packet, depth) if depth else O.decode(packet), f"{kind} {i}")

"""Headers gathered on the device: more frames than one launch takes, frames
cut in the frame header, in a picture header and between pictures, and sizes
that point past the data give what the host path gives."""

import numpy as np
import pytest

import rivet_prores_b200 as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 64, 65, 130])
def test_gathered_headers_plan_as_the_host_does(n):
    import torch

    base = []
    for interlace in range(3):
        p = O.test_frame(48, 32, 2, 10, 12, interlace)
        p.interlace = interlace
        k, msg, packet = O.encode(O.Config(3, luma_matrix=bytes([4] * 64) if interlace else None), p)
        assert k == O.OK, msg
        base.append(packet)
    rng = np.random.Generator(np.random.PCG64(n))
    frames = []
    for i in range(n):
        f = bytearray(base[i % 3])
        if i % 4 == 1:
            f = f[:int(rng.integers(0, len(f)))]  # cut anywhere, headers included
        elif i % 4 == 2:
            at = int(rng.choice([0, 1, 2, 3, 8, 9, 20, 29, 30, 31, 32, 33, 34]))
            f[at] = int(rng.integers(0, 256))
        elif i % 4 == 3 and i % 3:
            f[8 + 20 + 64 + 1:8 + 20 + 64 + 5] = int(rng.integers(0, 2 * len(f))).to_bytes(4, "big")  # picture_size
        frames.append(bytes(f))
    spans, at = [], 0
    for f in frames:
        spans.append((at, len(f)))
        at += len(f)
    data = torch.frombuffer(bytearray(b"".join(frames) + b"\0"), dtype=torch.uint8).cuda()
    got = P.Decoder.new().decode_device(data, spans, lambda k: torch.empty(k, dtype=torch.int16, device="cuda"))
    want = P.Decoder.new().decode_batch(frames)
    for i, (g, w) in enumerate(zip(got, want)):
        if isinstance(w, P.Error):
            assert type(g) is type(w) and g.message == w.message, (i, g, w)
        else:
            assert not isinstance(g, P.Error), (i, g)
            assert np.array_equal(g.data.cpu().numpy().view(np.uint16), w.data), i

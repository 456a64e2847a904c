"""The warp-per-32-blocks transform against the oracle, at the edges of how
slices are shared out to warps: every nominal slice width in both chroma
formats (whole components, several components or several slices a warp),
row-end slices of every smaller width, groups with a slice left over, fields,
planes whose rows do not start on 16 bytes, rows of zeros next to full ones."""

import numpy as np
import pytest

import rivet_prores_b200 as P
from oracle import oracle as O
from tests.util import assert_decode_matches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chroma,profile", [(2, 3), (2, 0), (3, 4)])
@pytest.mark.parametrize("log2", range(4))
def test_every_share_out_of_blocks(chroma, profile, log2):
    packets, depths = [], (8, 10, 16)
    for i, (w, h) in enumerate([(240, 33), (233, 50), (119, 17), (16, 16), (41, 64)]):
        for kind in ("noise", "flat"):
            rng = np.random.Generator(np.random.PCG64([log2, chroma, i]))
            p = O.test_frame(w, h, chroma, 10, 12, 10 * log2 + i)
            p.interlace = i % 3
            if kind == "flat":
                p.data[:] = 300
                p.data[rng.integers(0, p.data.size, 5)] = 900
            else:
                p.data[:] = rng.integers(0, 1024, p.data.size)
            k, msg, packet = O.encode(O.Config(profile, log2_slice_mbs=log2), p)
            assert k == O.OK, msg
            packets.append(packet)
    for depth in depths:
        got = P.Decoder.with_bit_depth(depth).decode_batch(packets)
        for i, (g, packet) in enumerate(zip(got, packets)):
            assert_decode_matches(g, O.decode(packet, depth), f"packet {i} at {depth} bits")

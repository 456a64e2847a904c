"""A batch with more quantiser table sets than a grid has rows (65,535): every
frame with a matrix of its own, those on both sides of the line and at the ends
against the oracle."""

import numpy as np
import pytest

import rivet_prores_b200 as P
from oracle import oracle as O
from tests.util import to_config, to_frame

pytestmark = pytest.mark.gpu


def test_more_matrices_than_a_grid_has_rows():
    n = 65537
    pic = O.test_frame(16, 16, 2, 10, 12, 3)
    weights = np.random.Generator(np.random.PCG64(1)).integers(2, 64, (n, 64), dtype=np.uint8)
    frame = to_frame(pic)
    configs = [P.Config(P.Profile.Hq, luma_matrix=w.tobytes()) for w in weights]
    got = P.Encoder(configs[0]).encode_batch([frame] * n, configs)
    for i in (0, 1, 65534, 65535, 65536):
        k, msg, want = O.encode(O.Config(3, luma_matrix=weights[i].tobytes()), pic)
        assert k == O.OK, msg
        assert got[i] == want, i

"""Packets written where the caller wants them: the same bytes as in library
memory, from host and from device planes, and a caller without room gets an
error and nothing else."""

import ctypes

import numpy as np
import pytest

import rivet_prores_b200 as P
from rivet_prores_b200 import _abi
from oracle import oracle as O
from tests.util import to_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("give_up", [False, True])
def test_packets_land_in_the_callers_room(device, give_up):
    import torch

    pics = [O.test_frame(64 + 16 * i, 48, 2, 10, 12, i) for i in range(3)]
    want = [O.encode(O.Config(3), p)[2] for p in pics]
    frames = [to_frame(p) for p in pics]
    keep, n = [], len(frames)
    cfgs, ins = (_abi.Config_ * n)(), (_abi.Frame_ * n)()
    outs, status = (_abi.Buf_ * n)(), (ctypes.c_int * n)()
    for i, f in enumerate(frames):
        cfgs[i] = P.Config(P.Profile.Hq)._c()
        ins[i] = P._frame_to_c(f, keep)
        if device:
            keep.append(torch.from_numpy(f.data.view(np.int16)).cuda())
            ins[i].data = ctypes.cast(keep[-1].data_ptr(), ctypes.POINTER(ctypes.c_uint16))
    rooms = [(ctypes.c_uint8 * (len(w) + 8))() for w in want]

    def room(_, i, size):
        return None if give_up and i == 1 else ctypes.addressof(rooms[i])

    code = _abi.lib().prores_encode_into(P.context(0).handle, cfgs, ins, n, int(device), _abi.PACKET_ROOM(room), None,
                                         outs, status, None)
    if give_up:
        assert code == _abi.DEVICE and all(not outs[i].data for i in range(n))
        return
    assert code == _abi.OK
    for i, w in enumerate(want):
        assert outs[i].len == len(w) and bytes(rooms[i][:len(w)]) == w and bytes(rooms[i][len(w):]) == bytes(8)

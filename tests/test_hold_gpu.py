"""Packets left where they arrive: the library keeps them apart from every
other call until they are freed, and an exception that a signal's handler
raises during an encode leaves the call as it would any other."""

import ctypes
import signal
import time

import pytest

import rivet_prores_b200 as P
from rivet_prores_b200 import _abi
from oracle import oracle as O
from tests.util import to_config, to_frame

pytestmark = pytest.mark.gpu


class Stop(Exception):
    pass


@pytest.mark.parametrize("share", [0.2, 0.5, 0.8])
def test_a_handlers_exception_leaves_the_encode(share):
    pic = to_frame(O.test_frame(1920, 1080, 2, 10, 12, 1))
    encoder = P.Encoder(P.Config(P.Profile.Hq))
    want = encoder.encode_batch([pic] * 8)
    begun = time.perf_counter()
    assert encoder.encode_batch([pic] * 8) == want
    took = time.perf_counter() - begun

    def stop(*_):
        raise Stop

    before = signal.signal(signal.SIGALRM, stop)
    try:
        for _ in range(5):
            with pytest.raises(Stop):
                signal.setitimer(signal.ITIMER_REAL, share * took)
                encoder.encode_batch([pic] * 8)
                time.sleep(10 * took)  # not before the call's end
    finally:
        signal.setitimer(signal.ITIMER_REAL, 0)
        signal.signal(signal.SIGALRM, before)
    assert encoder.encode_batch([pic] * 8) == want


def test_held_packets_outlast_other_calls():
    pics = [O.test_frame(64 + 16 * i, 48, 2, 10, 12, i) for i in range(3)]
    want = [O.encode(O.Config(3), p)[2] for p in pics]
    keep, n = [], len(pics) + 1
    cfgs, ins = (_abi.Config_ * n)(), (_abi.Frame_ * n)()
    outs, status = (_abi.Buf_ * n)(), (ctypes.c_int * n)()
    for i, p in enumerate(pics + pics[:1]):
        cfgs[i] = to_config(O.Config(3))._c()
        ins[i] = P._frame_to_c(to_frame(p), keep)
    cfgs[3].log2_slice_mbs = 9  # refused by itself
    L, held = _abi.lib(), ctypes.c_void_p()
    assert L.prores_encode_hold(P.context(0).handle, cfgs, ins, n, 0, outs, status, None,
                                ctypes.byref(held)) == _abi.OK and held
    assert [P.Encoder(P.Config(P.Profile.Hq)).encode(to_frame(p)) for p in reversed(pics)] == want[::-1]
    assert list(status[:3]) == [_abi.OK] * 3 and status[3] == _abi.CONFIG and outs[3].len == 0
    assert [ctypes.string_at(outs[i].data, outs[i].len) for i in range(3)] == want
    L.prores_packets_free(held)
    L.prores_packets_free(None)
    assert L.prores_encode_hold(P.context(0).handle, cfgs, ins, -1, 0, outs, status, None,
                                ctypes.byref(held)) == _abi.CONFIG and not held

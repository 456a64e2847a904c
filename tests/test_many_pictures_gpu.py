"""Batches of many small pictures: at the sizes where the forward transform's
search for its picture takes another round, and where the bisection gives a
picture fewer threads, every packet is the oracle's, and the kernels' times grow
no faster than the pictures."""

import pytest

import rivet_prores_b200 as P
from oracle import oracle as O
from tests.util import to_config, to_frame

pytestmark = pytest.mark.gpu

KINDS = [(16, 16, 2, 3, 0), (48, 32, 2, 3, 1), (33, 20, 3, 4, 2), (150, 16, 2, 1, 0), (16, 50, 3, 5, 1)]


# 1.6 pictures a frame: 32, 1024 and past both; 296 and past it (1024 threads a
# picture, then 512), and enough for 64.
@pytest.mark.parametrize("n", [1, 20, 21, 185, 186, 640, 641, 3000])
def test_every_packet_of_many_small_frames(n):
    frames, configs, want = [], [], []
    for i, (w, h, chroma, profile, interlace) in enumerate(KINDS):
        p = O.test_frame(w, h, chroma, 10, 12, i)
        p.interlace = interlace
        c = O.Config(profile, log2_slice_mbs=i % 4)
        k, msg, packet = O.encode(c, p)
        assert k == O.OK, msg
        frames.append(to_frame(p))
        configs.append(to_config(c))
        want.append(packet)
    at = [i % len(KINDS) for i in range(n)]
    got = P.Encoder(configs[0]).encode_batch([frames[k] for k in at], [configs[k] for k in at])
    for i, (g, k) in enumerate(zip(got, at)):
        assert g == want[k], (i, g if isinstance(g, P.Error) else len(g))


def _times(frames, config, kernel):
    """The shortest of three runs of each launch of `kernel`, in ms."""
    job = P.EncodeJob(frames, config)
    runs = []
    for _ in range(4):
        job.launch()
        job.fetch(copy=False)
        runs.append([ms for name, ms in job.kernel_times() if name == kernel])
    job.close()
    return [min(ms) for ms in zip(*runs[1:])]


def test_the_transform_takes_time_in_proportion_to_its_pictures(monkeypatch):
    monkeypatch.setenv("PRORES_PROFILE_KERNELS", "1")
    frame = to_frame(O.test_frame(16, 16, 2, 10, 12, 1))
    config = P.Config(P.Profile.Hq)
    few, many = 8192, 65536
    ratio = _times([frame] * many, config, "k_fdct")[0] / _times([frame] * few, config, "k_fdct")[0]
    assert ratio < 2 * many / few  # a search from end to end: 40


def test_a_bisection_step_of_many_pictures_is_short(monkeypatch):
    monkeypatch.setenv("PRORES_PROFILE_KERNELS", "1")
    frame = to_frame(O.test_frame(16, 16, 2, 10, 12, 1))
    config = P.Config(P.Profile.Hq)
    ratio = sum(_times([frame] * 4096, config, "k_rc_step")) / sum(_times([frame] * 64, config, "k_rc_step"))
    assert ratio < 6  # 1024 threads for every picture: 12

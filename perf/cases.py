"""The calls that users of this codec make, as cases that can be timed and
compared.

A case is one direction (`dir`: encode or decode) through one of the public
entry points (`entry`):

  call    `Decoder.decode` / `Encoder.encode`, one frame, host buffers in and
          out: the crate's own API, where a frame's latency counts.
  device  `Decoder.decode_device` / `Encoder.encode_device`: bitstreams or
          planes that already lie in device memory (a GPU player, a renderer
          that writes ProRes), the whole call with its header reads, its
          descriptors and its statuses.
  job     `DecodeJob` / `EncodeJob`: a batch kept resident and run again as
          one CUDA-graph launch (transcoding and serving); the decoded planes
          stay in device memory, the packets are fetched to the host.

Pictures are what the benchmark uses: smooth cosines, sharp-edged rectangles
and Gaussian noise, clamped to the video range, coded at the profile's own
target. They are made on the GPU from the seed alone. All outputs are
samples and bytes, which have one right value, so there is no `exact`.
"""

import math
import random

import numpy as np
import torch

import rivet_prores_b200 as P
from rivet_prores_b200 import _abi
from rivet_prores_b200.workloads import MIXED_KINDS, matrix

UHD_SAMPLES = 3840 * 2160 * 2


def _case(name, entry, dir, frames, width, height, profile, depth=10, out_depth=0, interlace=0, slice_log2=3,
          alpha_bits=0, noise=12.0, matrices=False, mixed=False):
    return {"name": name, "entry": entry, "dir": dir, "frames": frames, "width": width, "height": height,
            "profile": profile, "depth": depth, "out_depth": out_depth, "interlace": interlace,
            "slice_log2": slice_log2, "alpha_bits": alpha_bits, "noise": noise, "matrices": matrices, "mixed": mixed}


def listed():
    return [
        # One standard-definition interlaced 422 HQ frame from bytes to planes:
        # the smallest call, where launches and waits are all there is.
        _case("call_decode_sd", "call", "decode", 1, 720, 486, 3, interlace=2),
        # One 1080p frame to 422 HQ bytes: a capture or an editor's export, a
        # frame at a time.
        _case("call_encode_hd", "call", "encode", 1, 1920, 1080, 3),
        # One UHD frame decoded where it lies: a player's next frame.
        _case("device_decode_uhd", "device", "decode", 1, 3840, 2160, 3),
        # One rendered UHD frame coded from device memory.
        _case("device_encode_uhd", "device", "encode", 1, 3840, 2160, 3),
        # 1080p 422 HQ batches: the benchmark's 1080p configuration (64 frames
        # a launch) for playback, a second of 30 frames for a transcode's
        # encode.
        _case("job_decode_hd64", "job", "decode", 64, 1920, 1080, 3),
        _case("job_encode_hd30", "job", "encode", 30, 1920, 1080, 3),
        # The headline workload, UHD 422 HQ: 32 frames decoded through the
        # device-memory call, a second of 30 encoded as a resident batch.
        _case("device_decode_uhd32", "device", "decode", 32, 3840, 2160, 3),
        _case("job_encode_uhd30", "job", "encode", 30, 3840, 2160, 3),
        # UHD 4444 XQ: 12 bits, a 16-bit alpha plane, fields, loaded matrices
        # (the benchmark's mastering configuration), both ways.
        _case("device_decode_4444xq", "device", "decode", 8, 3840, 2160, 5, depth=12, interlace=1, alpha_bits=16,
              matrices=True),
        _case("job_encode_4444xq", "job", "encode", 8, 3840, 2160, 5, depth=12, interlace=1, alpha_bits=16,
              matrices=True),
        # Frames of every kind in one batch, 720x486 fields to 4096x2160 4:4:4
        # with alpha, slices of 1 to 8 macroblocks: what a server collects.
        _case("device_decode_mixed", "device", "decode", 28, 0, 0, 0, mixed=True),
        _case("job_encode_mixed", "job", "encode", 28, 0, 0, 0, mixed=True),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    """Any entry, direction, profile, size from 64x48 to 4096x2304 (odd ones
    among them), field order, slice width, depth and alpha type; the batch
    fills what is left of the largest listed amount of samples."""
    entry = rng.choice(["call", "device", "device", "job", "job", "job"])
    direction = rng.choice(["encode", "decode"])
    profile = rng.randrange(6)
    width = _log_uniform(rng, 64, 4096)
    height = max(48, int(width * rng.uniform(0.4, 0.75)))
    most = 32 * UHD_SAMPLES // 2
    if entry == "call":
        most = 1920 * 1080 * 2
    elif entry == "device" and direction == "encode":
        most = 2 * UHD_SAMPLES
    alpha = rng.choice([0, 0, 8, 16]) if profile >= 4 else 0
    if alpha:
        most //= 4
    per_frame = width * height * (3 if profile >= 4 else 2) + (width * height if alpha else 0)
    if entry == "call":
        while per_frame > most:
            width, height = max(64, width // 2), max(48, height // 2)
            per_frame = width * height * (3 if profile >= 4 else 2) + (width * height if alpha else 0)
    top = max(1, min(30 if direction == "encode" else 64, most // per_frame))
    frames = 1 if entry == "call" else _log_uniform(rng, 1, top)
    c = _case("", entry, direction, frames, width, height, profile,
              depth=rng.choice([8, 10, 10, 12, 16]), out_depth=rng.choice([0, 0, 0, 8, 12, 16]),
              interlace=rng.choice([0, 0, 1, 2]), slice_log2=rng.choice([3, 3, 2, 1, 0]), alpha_bits=alpha,
              noise=rng.choice([2.0, 6.0, 12.0, 20.0]), matrices=rng.random() < 0.25)
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs


def _frames_of(case):
    """(width, height, profile, depth, interlace, log2 slice mbs, alpha bits)
    of each frame of the case."""
    if not case["mixed"]:
        return [(case["width"], case["height"], P.Profile(case["profile"]), case["depth"],
                 P.Interlace(case["interlace"]), case["slice_log2"], case["alpha_bits"])] * case["frames"]
    out = []
    for i in range(case["frames"]):
        w, h, _, depth, profile, interlace, alpha = MIXED_KINDS[i % len(MIXED_KINDS)]
        out.append((w, h, profile, depth, interlace, (i // len(MIXED_KINDS) + i) % 4, 16 if alpha else 0))
    return out


def _plane(h, w, rng, gen, hi, noise):
    """Cosines, rectangles and noise at 10-bit scale (a float32 device plane)."""
    y = torch.arange(h, dtype=torch.float32, device="cuda")
    x = torch.arange(w, dtype=torch.float32, device="cuda")
    waves = [(rng.uniform(0, 0.05), rng.uniform(0, 0.05), rng.uniform(0, 150.0), rng.uniform(0, 2 * math.pi))
             for _ in range(8)]
    fx, fy, amp, phase = (torch.tensor(v, device="cuda")[:, None] for v in zip(*waves))
    ax, by = 2 * math.pi * fx * x + phase, 2 * math.pi * fy * y
    v = torch.cat([torch.cos(by), torch.sin(by)]).T @ torch.cat([amp * torch.cos(ax), -amp * torch.sin(ax)]) + 512.0
    for _ in range(16):
        x0, x1 = sorted(rng.randrange(w + 1) for _ in range(2))
        y0, y1 = sorted(rng.randrange(h + 1) for _ in range(2))
        v[y0:y1, x0:x1] = rng.uniform(64.0, 940.0)
    v += noise * torch.randn((h, w), generator=gen, device="cuda")
    return v.round_().clamp_(64.0, hi)


def _alpha(h, w, rng, gen):
    """Soft-edged ellipses over a clear background, with sensor noise."""
    y = torch.arange(h, dtype=torch.float32, device="cuda")[:, None]
    x = torch.arange(w, dtype=torch.float32, device="cuda")
    a = torch.zeros((h, w), device="cuda")
    for _ in range(4):
        cx, cy = rng.uniform(0, w), rng.uniform(0, h)
        rx, ry = rng.uniform(0.1, 0.4) * w, rng.uniform(0.1, 0.4) * h
        d = torch.sqrt(((x - cx) / rx) ** 2 + ((y - cy) / ry) ** 2)
        a = torch.maximum(a, ((1.0 - d) * 8.0).clamp(0.0, 1.0))
    a = a * 65535.0 + 200.0 * torch.randn((h, w), generator=gen, device="cuda")
    return a.round_().clamp_(0.0, 65535.0).to(torch.int32)


def _as_samples(v):
    """u16 samples as int16 bit patterns (torch's packed sample type here)."""
    return v.to(torch.int32).to(torch.int16).reshape(-1)


def _device_frames(case, seed):
    """The case's pictures in device memory, and each one's Config."""
    rng = random.Random(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    frames, configs = [], []
    for i, (w, h, profile, depth, interlace, log2, alpha_bits) in enumerate(_frames_of(case)):
        chroma = profile.chroma()
        cw = -(-w // chroma.subsampling()[0])
        planes = []
        for k, pw in enumerate((w, cw, cw)):
            v = _plane(h, pw, rng, gen, 940.0 if k == 0 else 960.0, case["noise"])
            planes.append(_as_samples(v * 2.0 ** (depth - 10) if depth >= 10 else (v / 4.0).round_()))
        alpha = None
        if alpha_bits:
            alpha = _as_samples(_alpha(h, w, rng, gen) >> (16 - depth))
        frames.append(P.DeviceFrame(w, h, depth, chroma, interlace, P.Metadata(), torch.cat(planes), alpha))
        loaded = {"luma_matrix": matrix(seed + i), "chroma_matrix": matrix(seed + i + 100)} if case["matrices"] else {}
        configs.append(P.Config(profile, log2_slice_mbs=log2,
                                alpha={0: P.AlphaType.None_, 8: P.AlphaType.Bits8, 16: P.AlphaType.Bits16}[alpha_bits],
                                **loaded))
    torch.cuda.synchronize()
    return frames, configs


def _host_frame(f):
    out = P.Frame.new(f.width, f.height, f.chroma, f.bit_depth)
    out.interlace = f.interlace
    out.data = f.data.cpu().numpy().view(np.uint16)
    out.alpha = None if f.alpha is None else f.alpha.cpu().numpy().view(np.uint16)
    return out


def _checked(results):
    for r in results:
        if isinstance(r, P.Error):
            raise r
    return results


class _DeviceArray:
    """int16 device memory at `ptr`, for torch.as_tensor."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i2", "data": (ptr, False), "strides": None,
                                         "version": 3}


class _FramePool:
    """A player's output surfaces: one device buffer, handed out frame by
    frame at 256-byte steps, used again for the next batch."""

    def __init__(self, samples):
        self.buffer = torch.zeros(samples, dtype=torch.int16, device="cuda")
        self.used = 0

    def __call__(self, n):
        at = self.used
        self.used = at + (n + 127) // 128 * 128
        return self.buffer[at:at + n]


_STREAM = []


def _stream():
    """The program's stream (one, as a program has for its codec work)."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0]


def _packet_length(frame, config):
    """The length of the two views _both_ends gives of a packet: packets come
    to between once and twice this (just under the profile's target, and the
    lossless alpha on top: up to 18 bits a noisy 16-bit value). A small
    packet's is well above what it can come to."""
    target = config.profile.target_frame_bytes(frame.width, frame.height)
    alpha = 0 if frame.alpha is None else frame.width * frame.height
    if target + 2 * alpha < 65536:
        return 4 * target + 3 * alpha + 65536
    return target * 3 // 4 + (alpha if config.alpha is P.AlphaType.Bits16 else alpha * 2 // 5)


def _both_ends(packet, n):
    """A whole packet in two views of n bytes (its first and its last n), so
    that packets of any length have outputs of one shape and none is copied;
    a packet shorter than n is copied into n bytes."""
    a = np.frombuffer(packet, np.uint8)
    if a.size > 2 * n:
        raise RuntimeError(f"a packet of {a.size} bytes, more than {2 * n}")
    if a.size >= n:
        return [a[:n], a[a.size - n:]]
    padded = np.zeros(n, np.uint8)
    padded[:a.size] = a
    return [padded, padded]


def prepare(case, seed):
    entry, direction = case["entry"], case["dir"]
    frames, configs = _device_frames(case, seed)
    state = {"entry": entry, "dir": direction, "lengths": [_packet_length(f, c) for f, c in zip(frames, configs)]}
    if direction == "encode":
        if entry == "device":
            return {**state, "encoder": P.Encoder(configs[0]), "frames": frames, "configs": configs}
        host = [_host_frame(f) for f in frames]
        if entry == "call":
            return {**state, "encoder": P.Encoder(configs[0]), "frame": host[0]}
        return {**state, "job": P.EncodeJob(host, configs)}
    packets = _checked(P.Encoder(configs[0]).encode_device(frames, configs))
    depth = case["out_depth"] or None
    if entry == "call":
        return {**state, "decoder": P.Decoder(depth), "packet": packets[0]}
    if entry == "device":
        data = torch.frombuffer(bytearray(b"".join(packets)), dtype=torch.uint8).cuda()
        spans, at = [], 0
        for p in packets:
            spans.append((at, len(p)))
            at += len(p)
        room = sum((f.data.numel() + 127) // 128 * 128 for f in frames)
        room += sum((f.alpha.numel() + 127) // 128 * 128 for f in frames if f.alpha is not None)
        return {**state, "decoder": P.Decoder(depth), "data": data, "spans": spans, "pool": _FramePool(room)}
    job = P.DecodeJob(packets, depth)
    # The batch's planes lie one frame after another, its alpha planes too.
    planes = []
    for k, numels in enumerate(([f.data.numel() for f in frames],
                                [f.alpha.numel() for f in frames if f.alpha is not None])):
        if numels:
            ptrs = (P.ctypes.POINTER(P.ctypes.c_uint16)(), P.ctypes.POINTER(P.ctypes.c_uint16)())
            if _abi.lib().prores_decode_job_planes(job.handle, 0, P.ctypes.byref(ptrs[0]), P.ctypes.byref(ptrs[1])):
                raise RuntimeError(_abi.last_error())
            planes.append(torch.as_tensor(_DeviceArray(P.ctypes.cast(ptrs[k], P.ctypes.c_void_p).value, sum(numels)),
                                          device="cuda"))
    return {**state, "job": job, "planes": planes}


def run(state):
    entry = state["entry"]
    if state["dir"] == "encode":
        if entry == "call":
            packets = [state["encoder"].encode(state["frame"])]
        elif entry == "device":
            packets = state["encoder"].encode_device(state["frames"], state["configs"], stream=_stream())
        else:
            state["job"].launch(_stream(), graph=True)
            packets = state["job"].fetch(_stream(), copy=False)
        views = [v for p, n in zip(_checked(packets), state["lengths"]) for v in _both_ends(p, n)]
        return [np.array([len(p) for p in packets])] + views
    if entry == "call":
        f = state["decoder"].decode(state["packet"])
        return [f.data] if f.alpha is None else [f.data, f.alpha]
    if entry == "device":
        state["pool"].used = 0
        _checked(state["decoder"].decode_device(state["data"], state["spans"], state["pool"], stream=_stream()))
        return state["pool"].buffer
    state["job"].launch(_stream(), graph=True)
    return state["planes"]


def work(case):
    """Every sample read or written once, every packet (the profile's target,
    and two bytes for each alpha value, about what noisy alpha takes) once;
    two 8-point transforms of 64 multiplies and adds a block row and column."""
    samples = packet = 0
    for w, h, profile, _, _, _, alpha_bits in _frames_of(case):
        cw = -(-w // profile.chroma().subsampling()[0])
        n = h * (w + 2 * cw)
        samples += n
        packet += profile.target_frame_bytes(w, h)
        if alpha_bits:
            samples += w * h
            packet += alpha_bits // 8 * w * h
    return {"bytes": packet + 2 * samples, "flops": 32 * samples}

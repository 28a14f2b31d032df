"""The work that is timed: decoding, encoding and training as programs call them.

`listed()` names the cases, `draw()` gives more of the same ranges. A case is
a dict of plain values; `prepare()` makes what a program holds before the call
(inputs on the GPU, a handle, weights), `run()` is one pass through the public
entry points, `exact()` the same results in 64 bits in plain torch where they
are computed numbers, `work()` the bytes and operations of one pass.

Kinds of cases:
  frame    one frame per call on host memory (the reference's decode(float*))
  plain    a device batch through the bit-exact normalized min-sum decoder
  learned  a device batch through the learned min-sum decoder in fp32
  half     the same decoder in packed binary16
  mixed    a device batch whose frames are of any of the 114 codes
  train    loss and weight gradient of one generated batch
  encode   a device batch through the encoder
  host     a host batch (pinned buffers) copied in, decoded, hard bits copied back
"""
import math

import numpy as np
import torch

import wimax_ldpc_lib_b200 as wl
from wimax_ldpc_lib_b200 import mixed_batch

CAP = 10            # the reference's iteration cap
TRAINED = 8         # iterations the shipped weights were trained with
MIB = 1 << 20

# Eb/N0 at z = 96 just right of each rate's waterfall, where a link runs
EBNO = (2.25, 2.75, 2.75, 3.25, 3.25, 4.0)
RATE = (1 / 2, 2 / 3, 2 / 3, 3 / 4, 3 / 4, 5 / 6)

# IEEE 802.16e base matrices, one text per base row: block column:shift at z = 96
BASE = (
    (   # rate 1/2
        "1:94 2:73 8:55 9:83 12:7 13:0",
        "1:27 5:22 6:79 7:9 11:12 13:0 14:0",
        "3:24 4:22 5:81 7:33 11:0 14:0 15:0",
        "0:61 2:47 8:65 9:25 15:0 16:0",
        "2:39 6:84 9:41 10:72 16:0 17:0",
        "4:46 5:40 7:82 11:79 12:0 17:0 18:0",
        "2:95 3:53 9:14 10:18 18:0 19:0",
        "1:11 2:73 6:2 9:47 19:0 20:0",
        "0:12 4:83 5:24 7:43 11:51 20:0 21:0",
        "5:94 7:59 10:70 11:72 21:0 22:0",
        "2:7 3:65 8:39 9:49 22:0 23:0",
        "0:43 5:66 7:41 11:26 12:7 23:0",
    ),
    (   # rate 2/3A
        "0:3 1:0 4:2 5:0 7:3 8:7 10:1 11:1 16:1 17:0",
        "2:1 4:36 7:34 8:10 11:18 12:2 14:3 15:0 17:0 18:0",
        "2:12 3:2 5:15 7:40 9:3 11:15 13:2 14:13 18:0 19:0",
        "2:19 3:24 5:3 6:0 8:6 10:17 14:8 15:39 19:0 20:0",
        "0:20 2:6 5:10 6:29 9:28 11:14 13:38 16:0 20:0 21:0",
        "2:10 4:28 5:20 8:8 10:36 12:9 14:21 15:45 21:0 22:0",
        "0:35 1:25 3:37 5:21 8:5 11:0 13:4 14:20 22:0 23:0",
        "1:6 2:6 6:4 8:14 9:30 11:3 12:36 14:14 16:1 23:0",
    ),
    (   # rate 2/3B
        "0:2 2:19 4:47 6:48 8:36 10:82 12:47 14:15 16:95 17:0",
        "1:69 3:88 5:33 7:3 9:16 11:37 13:40 15:48 17:0 18:0",
        "0:10 2:86 4:62 6:28 8:85 10:16 12:34 14:73 18:0 19:0",
        "1:28 3:32 5:81 7:27 9:88 11:5 13:56 15:37 19:0 20:0",
        "0:23 2:29 4:15 6:30 8:66 10:24 12:50 14:62 20:0 21:0",
        "1:30 3:65 5:54 7:14 9:0 11:30 13:74 15:0 21:0 22:0",
        "0:32 2:0 4:15 6:56 8:85 10:5 12:6 14:52 16:0 22:0 23:0",
        "1:0 3:47 5:13 7:61 9:84 11:55 13:78 15:41 16:95 23:0",
    ),
    (   # rate 3/4A
        "0:6 1:38 2:3 3:93 7:30 8:70 10:86 12:37 13:38 14:4 15:11 17:46 18:48 19:0",
        "0:62 1:94 2:19 3:84 5:92 6:78 8:15 11:92 13:45 14:24 15:32 16:30 19:0 20:0",
        "0:71 2:55 4:12 5:66 6:45 7:79 9:78 12:10 14:22 15:55 16:70 17:82 20:0 21:0",
        "0:38 1:61 3:66 4:9 5:73 6:47 7:64 9:39 10:61 11:43 16:95 17:32 18:0 21:0 22:0",
        "4:32 5:52 6:55 7:80 8:95 9:22 10:6 11:51 12:24 13:90 14:44 15:20 22:0 23:0",
        "1:63 2:31 3:88 4:20 8:6 9:40 10:56 11:16 12:71 13:53 16:27 17:26 18:48 23:0",
    ),
    (   # rate 3/4B
        "1:81 3:28 6:14 7:25 8:17 11:85 12:29 13:52 14:78 15:95 16:22 17:92 18:0 19:0",
        "0:42 2:14 3:68 4:32 9:70 10:43 11:11 12:36 13:40 14:33 15:57 16:38 17:24 19:0 20:0",
        "2:20 5:63 6:39 8:70 9:67 11:38 12:4 13:72 14:47 15:29 16:60 17:5 18:80 20:0 21:0",
        "0:64 1:2 4:63 7:3 8:51 10:81 11:15 12:94 13:9 14:85 15:36 16:14 17:19 21:0 22:0",
        "1:53 2:60 3:80 5:26 6:75 11:86 12:77 13:1 14:3 15:72 16:60 17:25 22:0 23:0",
        "0:77 4:15 5:28 7:35 9:72 10:30 11:68 12:85 13:84 14:26 15:64 16:11 17:89 18:0 23:0",
    ),
    (   # rate 5/6
        "0:1 1:25 2:55 4:47 5:4 7:91 8:84 9:8 10:86 11:52 12:82 13:33 14:5 15:0 16:36 17:20 18:4 19:77 20:80 21:0",
        "1:6 3:36 4:40 5:47 6:12 7:79 8:47 10:41 11:21 12:12 13:71 14:14 15:72 16:0 17:44 18:49 19:0 20:0 21:0 22:0",
        "0:51 1:81 2:83 3:4 4:67 6:21 8:31 9:24 10:91 11:61 12:81 13:9 14:86 15:78 16:60 17:88 18:67 19:15 22:0 23:0",
        "0:50 2:50 3:15 5:36 6:13 7:10 8:11 9:20 10:53 11:90 12:29 13:92 14:57 15:30 16:84 17:92 18:11 19:66 20:80 23:0",
    ),
)


def base_rows(rate, z):
    """[(block columns, shifts at z)] of the code's base rows."""
    rows = []
    for text in BASE[rate]:
        pairs = [tuple(int(x) for x in p.split(":")) for p in text.split()]
        rows.append(([c for c, _ in pairs],
                     [s if s == 0 else s % z if rate == 1 else s * z // 96 for _, s in pairs]))
    return rows


def edges(rate, z):
    return z * sum(len(text.split()) for text in BASE[rate])


def ebno(rate, z):
    """A working Eb/N0 for the code: shorter codes need up to half a dB more."""
    return round(EBNO[rate] + (96 - z) * 0.0065, 3)


def case(name, kind, rate=0, z=96, frames=1, soft=False, cap=CAP):
    c = {"kind": kind, "rate": rate, "z": z, "frames": frames, "ebno": ebno(rate, z), "soft": soft, "cap": cap}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a program ported from the reference: decode(float*) called per received frame
        case("frame_r12_z96", "frame"),
        # the code blocks of one radio frame, soft output for the next stage
        case("burst_r34a_z52", "plain", rate=3, z=52, frames=96, soft=True),
        # a base station's or simulator's batch of the longest rate-1/2 code, bits only
        case("plain_r12_z96", "plain", frames=65536),
        # a ragged batch of a code whose z is no multiple of 32, soft output
        case("plain_r23b_z44", "plain", rate=2, z=44, frames=20011, soft=True),
        # the learned decoder on the benchmark's code
        case("learned_r12_z96", "learned", frames=65536),
        # high rate, wide check rows, ragged, soft output
        case("learned_r56_z60", "learned", rate=5, z=60, frames=30011, soft=True),
        # highest-throughput option: packed binary16
        case("half_r12_z96", "half", frames=131072),
        case("half_r34a_z36", "half", rate=3, z=36, frames=40003, soft=True),
        # a base station's uplink: every frame of its own code and quality
        case("mixed_65536", "mixed", frames=65536),
        # one training step of the learned decoder at the training script's batch
        case("train_r12_z96", "train", frames=4096),
        # a transmitter's or simulator's batch
        case("encode_r12_z96", "encode", frames=262144),
        # host buffers in, hard bits out, through the copy pipeline
        case("host_r12_z96", "host", frames=16384),
    ]


def draw(rng):
    kind = rng.choice(("plain", "plain", "plain", "learned", "learned", "learned", "half", "half", "mixed", "train",
                       "encode", "frame"))
    rate, z = rng.randrange(6), rng.choice(wl.Z_VALUES)
    lo, hi = {"frame": (1, 1), "mixed": (1024, 65536), "train": (64, 4096), "encode": (512, 262144)}.get(kind, (48, 65536))
    frames = round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))
    if kind == "train":
        rate = rng.choice((0, 1, 2, 3, 5))
    if kind == "encode":
        rate = rng.choice((0, 1, 2, 3, 5))
    soft = rng.random() < 0.4 and kind in ("plain", "learned", "half")
    cap = rng.choice((CAP, CAP, 5, 8, 20)) if kind in ("plain", "learned", "half") else CAP
    c = case(None, kind, rate, z, frames, soft, cap)
    return dict(c, ebno=round(c["ebno"] + rng.uniform(-0.2, 0.5), 3))


def inputs(c, seed):
    """(codewords, LLRs) of frames x n on the GPU: random codewords, BPSK, white noise."""
    n = 24 * c["z"]
    cw = torch.empty((c["frames"], n), dtype=torch.uint8, device="cuda")
    llr = torch.empty((c["frames"], n), dtype=torch.float32, device="cuda")
    make = wl.framegen_nullspace_device if c["rate"] == 4 else wl.framegen_device
    make(c["rate"], c["z"], seed, 0, c["frames"], c["ebno"], codeword=cw, llr=llr)
    return cw, llr


def learned(c, precision=wl.LMS_F32):
    _, weights, _ = wl.learned_weights(c["rate"], c["z"])
    return wl.LearnedDecoder(c["rate"], c["z"], TRAINED, weights, None if c["kind"] == "train" else c["cap"], precision)


def prepare(c, seed):
    kind, rate, z, frames = c["kind"], c["rate"], c["z"], c["frames"]
    n = 24 * z
    s = {"case": c, "seed": seed}
    if kind == "frame":
        s["dec"] = wl.Decoder(rate, z, c["cap"])
        s["llr"] = inputs(c, seed)[1][0].cpu().numpy()
    elif kind in ("plain", "learned", "half"):
        s["dec"] = (wl.Decoder(rate, z, c["cap"]) if kind == "plain" else
                    learned(c, wl.LMS_F16X2 if kind == "half" else wl.LMS_F32))
        s["llr"] = inputs(c, seed)[1]
        s["hard"] = torch.empty((frames, n), dtype=torch.int8, device="cuda")
        s["post"] = torch.empty_like(s["llr"]) if c["soft"] else None
        s["status"] = torch.empty(frames, dtype=torch.int32, device="cuda")
    elif kind == "mixed":
        s["dec"] = wl.MixedDecoder(c["cap"])
        s["variants"], s["offsets"], s["llr"], _, _ = mixed_batch.build_batch(frames, seed=seed, ebno=(1.0, 4.0))
        # room for frames of the longest code: the batch's own length depends on its codes
        s["hard"] = torch.zeros(frames * 2304, dtype=torch.int8, device="cuda")
        s["status"] = torch.empty(frames, dtype=torch.int32, device="cuda")
    elif kind == "train":
        s["dec"] = learned(c)
        s["grad"] = torch.empty(s["dec"].grad_size(), dtype=torch.float32, device="cuda")
        s["loss"] = torch.empty(1, dtype=torch.float32, device="cuda")
    elif kind == "encode":
        s["enc"] = wl.Encoder(rate, z)
        g = torch.Generator(device="cuda").manual_seed(seed)
        s["info"] = torch.randint(0, 2, (frames, s["enc"].k), dtype=torch.uint8, device="cuda", generator=g)
        s["cw"] = torch.empty((frames, n), dtype=torch.uint8, device="cuda")
    elif kind == "host":
        s["dec"] = wl.Decoder(rate, z, c["cap"])
        s["llr"] = torch.empty((frames, n), dtype=torch.float32, pin_memory=True).copy_(inputs(c, seed)[1])
        s["hard"] = torch.empty((frames, n), dtype=torch.int8, pin_memory=True)
        s["errors"] = torch.empty(frames, dtype=torch.int32, pin_memory=True)
        s["status"] = torch.empty(frames, dtype=torch.int32, pin_memory=True)
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "frame":
        post, hard, failed, iterations = s["dec"].decode(s["llr"])
        return {"post": post, "hard": hard, "failed": failed, "iterations": iterations}
    if kind in ("plain", "learned", "half"):
        s["dec"].decode_device(s["llr"], s["hard"], s["post"], s["status"])
        return {"post": s["post"], "hard": s["hard"], "status": s["status"]}
    if kind == "mixed":
        s["dec"].decode_device(s["variants"], s["offsets"], s["llr"], s["hard"], None, s["status"])
        return {"hard": s["hard"], "status": s["status"]}
    if kind == "train":
        s["dec"].step_grad(c["frames"], c["ebno"] - 1.25, c["ebno"] + 0.75, s["seed"], 0, s["grad"], s["loss"])
        return {"grad": s["grad"], "loss": s["loss"]}
    if kind == "encode":
        s["enc"].encode_device(s["info"], s["cw"])
        return {"codeword": s["cw"]}
    s["dec"].decode_host_hard_into(s["llr"], s["hard"], s["errors"], s["status"])
    return {"hard": s["hard"], "errors": s["errors"], "status": s["status"]}


def work(c):
    """Every input read once and every output written once. Operations: per
    edge and iteration a subtraction, two comparisons, a multiplication, a
    subtraction, a comparison and an addition (four iterations, about the mean
    at these Eb/N0); a training step runs them three times (forward,
    recomputed forward, backward) for the trained iterations."""
    rate, z, frames, kind = c["rate"], c["z"], c["frames"], c["kind"]
    n, e = 24 * z, edges(rate, z)
    if kind == "mixed":
        n, e = 24 * 60, sum(edges(r, 60) for r in range(6)) / 6
    if kind == "encode":
        return {"bytes": frames * n * (1 + RATE[rate]), "flops": 0}
    if kind == "train":
        return {"bytes": 4 * 3 * TRAINED * e / z * 2, "flops": frames * e * TRAINED * 7 * 3}
    out = n + 4 + (4 * n if c["soft"] or kind == "frame" else 0)
    return {"bytes": frames * (4 * n + out), "flops": frames * e * 4 * 7}


def layered(rows, z, llr, scale, offset, iterations, clamp, stop):
    """Layered min-sum in 64 bits over llr (frames x n). scale, offset:
    [iteration][base row][block column]; clamp bounds the minima. Returns the
    posteriors after every iteration; with stop, the final ones, a frame
    staying as it is from its first zero syndrome on."""
    dev = llr.device
    r = torch.arange(z, device=dev)
    at = [torch.stack([col * z + (r + s) % z for col, s in zip(*row)], 1) for row in rows]   # z x degree
    post, seen = llr, []
    msgs = [torch.zeros((llr.shape[0],) + a.shape, dtype=torch.float64, device=dev) for a in at]

    def fails(p):
        bits = p >= 0
        return torch.stack([(bits[:, a].sum(2) % 2 == 1).any(1) for a in at]).any(0)

    going = fails(post) if stop else None
    for t in range(iterations):
        if stop and not bool(going.any()):
            break
        new, before = post, post
        w = min(t, scale.shape[0] - 1)
        for i, (a, (cols, _)) in enumerate(zip(at, rows)):
            x = new[:, a] - msgs[i]
            low, first = x.abs().topk(2, dim=2, largest=False)
            edge = torch.arange(a.shape[1], device=dev)
            mu = torch.where(edge == first[..., :1], low[..., 1:], low[..., :1]).clamp(max=clamp)
            neg = (x < 0).long()
            odd = (neg.sum(2, keepdim=True) + neg + a.shape[1]) % 2
            msgs[i] = (1 - 2 * odd) * torch.relu(scale[w, i, cols] * mu - offset[w, i, cols])
            new = new.index_copy(1, a.reshape(-1), (x + msgs[i]).flatten(1))
        post = torch.where(going[:, None], new, before) if stop else new
        if stop:
            going = going & fails(post)
        seen.append(post)
    return post if stop else seen


def exact(c, seed):
    kind, rate, z = c["kind"], c["rate"], c["z"]
    rows = base_rows(rate, z)
    if kind == "train":
        n = 24 * z
        cw = torch.empty((c["frames"], n), dtype=torch.uint8, device="cuda")
        llr = torch.empty((c["frames"], n), dtype=torch.float32, device="cuda")
        make = wl.framegen_nullspace_device if rate == 4 else wl.framegen_device
        make(rate, z, seed, 0, c["frames"], c["ebno"] - 1.25, c["ebno"] + 0.75, codeword=cw, llr=llr)
        _, weights, _ = wl.learned_weights(rate, z)
        w = torch.tensor(weights, dtype=torch.float64, device="cuda", requires_grad=True)
        total = 0.0
        for f in range(0, c["frames"], 512):
            seen = layered(rows, z, llr[f:f + 512].double(), w[0], w[1], TRAINED, math.inf, False)
            sign = 1.0 - 2.0 * cw[f:f + 512].double()
            loss = sum(torch.nn.functional.softplus(sign * p, threshold=700.0).sum() for p in seen)
            loss = loss / (TRAINED * n * c["frames"])
            loss.backward()
            total += loss.detach()
        keep = torch.zeros(weights.shape[1:], dtype=torch.bool, device="cuda")
        for i, (cols, _) in enumerate(rows):
            keep[:, i, cols] = True
        return {"grad": w.grad[:, keep].reshape(-1), "loss": total.reshape(1)}
    values = c["frames"] * 24 * z
    if kind == "frame" or (c["soft"] and kind in ("plain", "learned") and values <= 64 * MIB):
        llr = inputs(c, seed)[1].double()
        if kind == "learned":
            w = torch.tensor(wl.learned_weights(rate, z)[1], dtype=torch.float64, device="cuda")
            scale, offset, clamp = w[0], w[1], math.inf
        else:
            scale = torch.full((1, 12, 24), 0.815, dtype=torch.float64, device="cuda")
            offset, clamp = torch.zeros_like(scale), 10000.0
        post = torch.cat([layered(rows, z, part, scale, offset, c["cap"], clamp, True) for part in llr.split(4096)])
        if kind == "frame":
            return {"post": post[0].cpu().numpy(), "hard": None, "failed": None, "iterations": None}
        return {"post": post, "hard": None, "status": None}
    # bits and counts, or binary16 arithmetic that is fixed operation by operation
    return None

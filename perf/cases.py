"""The work the encoder is timed on, through its public entry points.

Each case is one call that a program using this package makes:

  encode    one RGBA8 texture to ASTC blocks: secondaryInit + encode (host buffers) or
            encode_device (device buffers), by the full search (the reference's semantics or
            the repaired ones) or the learned proposal search, with or without the optional
            void-extent and dual-plane encodings
  batch     many textures of mixed sizes and footprints in one call: encode_batch
  mipchain  a texture's whole mip chain to .astc containers: mipchain.encode_mip_chain_astc
  decode    ASTC blocks to RGBA8 (decode_device), or compared with the original texture for a
            PSNR (decode_error_device)
  train     one forward and backward pass of the proposal network: proposal.Trainer

A program keeps one encoder per configuration and encodes texture after texture with it, so
the encoders (and the stream their device calls go to) outlive a case's inputs here too.
Textures follow the package's synthetic generator (synth.py): value noise with hard-edged
rectangles and diagonal splits, opaque on the left half.
"""
import math

import numpy as np
import torch

import astc_implementation_b200 as ab
from astc_implementation_b200 import flop_model, mipchain, proposal

NETWORK_FOOTPRINTS = ((4, 4), (6, 6))

_ENCODE = {"kind": "encode", "search": "full", "fixed": False, "extend": False, "io": "host", "chunk": 0}


def _encode(**kw):
    return dict(_ENCODE, **kw)


def listed():
    return [
        # a thumbnail or a small mip level through the reference's own call: the smallest call,
        # where launches and the longest chain of one block count
        _encode(name="full_64x64_4x4", w=64, h=64, bx=4, by=4),
        # an ordinary texture by the full search, device to device inside an asset pipeline
        _encode(name="full_1024x1024_4x4_fixed", w=1024, h=1024, bx=4, by=4, fixed=True, io="device"),
        # the low-bit-rate footprints, with edges that are no multiple of the block
        _encode(name="full_1021x765_10x8", w=1021, h=765, bx=10, by=8),
        # a small UI texture by the proposal search
        _encode(name="prop_200x120_4x4", w=200, h=120, bx=4, by=4, search="proposal", fixed=True),
        # the headline benchmark's texture and settings, host to host from pinned memory
        _encode(name="prop_2048x2048_4x4", w=2048, h=2048, bx=4, by=4, search="proposal", fixed=True, io="pinned",
                chunk=262144),
        # the same at 6x6 with the default chunk, device to device, ragged edges
        _encode(name="prop_2047x2050_6x6", w=2047, h=2050, bx=6, by=6, search="proposal", fixed=True, io="device"),
        # the largest texture, default chunk
        _encode(name="prop_4096x4096_4x4", w=4096, h=4096, bx=4, by=4, search="proposal", fixed=True, io="device"),
        # the highest quality setting: proposal search, then void-extent and dual-plane blocks
        _encode(name="prop_ext_1024x1024_4x4", w=1024, h=1024, bx=4, by=4, search="proposal", fixed=True, extend=True,
                io="device"),
        # an asset import: many small textures, mixed footprints, host to host
        {"name": "batch_16_mixed", "kind": "batch", "count": 16, "min_side": 48, "max_side": 640},
        # an engine's texture import: the mip chain, from a host image to containers
        {"name": "mipchain_1024x1024_6x6", "kind": "mipchain", "w": 1024, "h": 1024, "bx": 6, "by": 6},
        # a texture upload without hardware decoding
        {"name": "decode_4096x4096_6x6", "kind": "decode", "w": 4096, "h": 4096, "bx": 6, "by": 6, "error": False},
        # training a network for one's own textures: one step's forward and backward pass at
        # the training driver's batch
        {"name": "train_4x4_2048", "kind": "train", "bx": 4, "by": 4, "rows": 2048},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["full", "proposal", "extend", "batch", "mipchain", "decode", "train"],
                       [30, 28, 10, 8, 8, 10, 6])[0]
    if kind == "full":
        bx, by = rng.choice(ab.VALID_FOOTPRINTS)
        return _encode(w=_log_int(rng, 16, 900), h=_log_int(rng, 16, 900), bx=bx, by=by, fixed=rng.random() < 0.5,
                       io=rng.choice(["host", "device"]))
    if kind == "proposal":
        bx, by = rng.choice(NETWORK_FOOTPRINTS)
        return _encode(w=_log_int(rng, 40, 4000), h=_log_int(rng, 40, 4000), bx=bx, by=by, search="proposal", fixed=True,
                       io=rng.choice(["host", "pinned", "device"]), chunk=rng.choice([0, 0, 262144]))
    if kind == "extend":
        bx, by = rng.choice(NETWORK_FOOTPRINTS)
        return _encode(w=_log_int(rng, 40, 1000), h=_log_int(rng, 40, 1000), bx=bx, by=by, search="proposal", fixed=True,
                       extend=True, io=rng.choice(["host", "device"]))
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(3, 20), "min_side": 48, "max_side": _log_int(rng, 96, 560)}
    if kind == "mipchain":
        bx, by = rng.choice(NETWORK_FOOTPRINTS)
        return {"kind": "mipchain", "w": _log_int(rng, 100, 1500), "h": _log_int(rng, 100, 1500), "bx": bx, "by": by}
    if kind == "decode":
        bx, by = rng.choice(NETWORK_FOOTPRINTS + ((8, 8), (12, 10)))
        top = 4000 if (bx, by) in NETWORK_FOOTPRINTS else 1000
        return {"kind": "decode", "w": _log_int(rng, 60, top), "h": _log_int(rng, 60, top), "bx": bx, "by": by,
                "error": rng.random() < 0.5}
    bx, by = rng.choice(NETWORK_FOOTPRINTS)
    return {"kind": "train", "bx": bx, "by": by, "rows": _log_int(rng, 128, 2048)}


# ------------------------------------------------------------ inputs

def _texture(w, h, seed):
    """(h, w, 4) uint8 on the GPU, by synth.make_texture's recipe."""
    rng = np.random.default_rng(seed)
    dev = torch.device("cuda")
    img = torch.zeros(4, h, w, dtype=torch.float32, device=dev)
    weight = 0.0
    for o in range(4):
        g = 2 ** (o + 2) + 1
        grid = torch.from_numpy(rng.random((1, 4, g, g)).astype(np.float32)).to(dev)
        img += torch.nn.functional.interpolate(grid, size=(h, w), mode="bilinear", align_corners=True)[0] * 0.5 ** o
        weight += 0.5 ** o
    img *= 255.0 / weight

    def box():
        x0, x1 = np.sort(rng.integers(0, w + 1, 2))
        y0, y1 = np.sort(rng.integers(0, h + 1, 2))
        colour = torch.from_numpy(rng.integers(0, 256, 3).astype(np.float32)).to(dev).view(3, 1, 1)
        return int(x0), int(x1), int(y0), int(y1), colour

    for _ in range(32):
        x0, x1, y0, y1, colour = box()
        img[:3, y0:y1, x0:x1] = colour
    for _ in range(16):
        x0, x1, y0, y1, colour = box()
        ang = math.radians(rng.choice([45.0, 135.0]) + rng.uniform(-15.0, 15.0))
        xx = torch.arange(x0, x1, dtype=torch.float32, device=dev) - (x0 + x1) / 2.0
        yy = torch.arange(y0, y1, dtype=torch.float32, device=dev) - (y0 + y1) / 2.0
        side = (xx * math.sin(ang))[None, :] - (yy * math.cos(ang))[:, None] > 0
        part = img[:3, y0:y1, x0:x1]
        part.copy_(torch.where(side[None], colour, part))
    img[3, :, : w // 2] = 255.0
    return img.round_().clamp_(0, 255).to(torch.uint8).permute(1, 2, 0).contiguous()


def _blocks(w, h, bx, by):
    return ((w + bx - 1) // bx) * ((h + by - 1) // by)


_encoders = {}
_networks = {}


def _network(bx, by):
    if (bx, by) not in _networks:
        _networks[bx, by] = proposal.load_weights(bx, by)
    return _networks[bx, by]


def _encoder(search, fixed, extend, chunk):
    """The program's encoder of one configuration, with the stream of its device calls."""
    key = (search, fixed, extend, chunk)
    if key not in _encoders:
        enc = ab.ASTCEncoder(device=torch.cuda.current_device(), fixed=fixed, void_extent=extend, dual_plane=extend,
                             chunk_blocks=chunk)
        enc.init()
        if search == "proposal":
            for bx, by in NETWORK_FOOTPRINTS:
                enc.set_proposal_net(_network(bx, by))
            enc.set_pruning(True)
        _encoders[key] = enc, torch.cuda.Stream()
    return _encoders[key]


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


def _prepare_encode(c, seed):
    enc, stream = _encoder(c["search"], c["fixed"], c["extend"], c["chunk"])
    img = _texture(c["w"], c["h"], seed)
    nbytes = 16 * _blocks(c["w"], c["h"], c["bx"], c["by"])
    s = {"kind": "encode", "enc": enc, "stream": stream, "size": (c["w"], c["h"], c["bx"], c["by"]), "io": c["io"]}
    if c["io"] == "device":
        s["image"], s["out"] = img, torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
    elif c["io"] == "pinned":
        s["keep"] = img.cpu().pin_memory(), torch.zeros(nbytes, dtype=torch.uint8).pin_memory()
        s["image"], s["out"] = s["keep"][0].numpy(), s["keep"][1].numpy()
    else:
        s["image"], s["out"] = img.cpu().numpy(), None
    return s


def _run_encode(s):
    enc = s["enc"]
    enc.secondaryInit(*s["size"])
    if s["io"] == "device":
        enc.encode_device(s["image"].data_ptr(), s["out"].data_ptr(), s["stream"].cuda_stream)
        return s["out"]
    return enc.encode(s["image"], s["out"])


_BATCH_FOOTPRINTS = ((4, 4), (6, 6), (8, 8))


def _batch_sizes(c):
    """Sides log-uniform per axis, footprints in turn; part of the case, not of its inputs."""
    rng = np.random.default_rng(1000 + c["count"])
    out = []
    for i in range(c["count"]):
        w, h = np.exp(rng.uniform(np.log(c["min_side"]), np.log(c["max_side"]), 2))
        out.append((int(w), int(h)) + _BATCH_FOOTPRINTS[i % 3])
    return out


def _prepare_batch(c, seed):
    enc, _ = _encoder("full", False, False, 0)
    tex = [(_texture(w, h, 1000 * seed + i).cpu().numpy(), bx, by) for i, (w, h, bx, by) in enumerate(_batch_sizes(c))]
    return {"kind": "batch", "enc": enc, "textures": tex}


def _run_batch(s):
    return s["enc"].encode_batch(s["textures"])


def _prepare_mipchain(c, seed):
    enc, _ = _encoder("proposal", True, False, 0)
    return {"kind": "mipchain", "enc": enc, "image": _texture(c["w"], c["h"], seed).cpu().numpy(), "foot": (c["bx"], c["by"])}


def _run_mipchain(s):
    files = mipchain.encode_mip_chain_astc(s["enc"], s["image"], *s["foot"])
    return [np.frombuffer(f, np.uint8) for f in files]


def _prepare_decode(c, seed):
    w, h, bx, by = c["w"], c["h"], c["bx"], c["by"]
    search = "proposal" if (bx, by) in NETWORK_FOOTPRINTS else "full"
    enc, stream = _encoder(search, True, False, 0)
    img = _texture(w, h, seed)
    blocks = torch.zeros(16 * _blocks(w, h, bx, by), dtype=torch.uint8, device="cuda")
    torch.cuda.current_stream().synchronize()  # the texture was made on another stream
    enc.secondaryInit(w, h, bx, by)
    enc.encode_device(img.data_ptr(), blocks.data_ptr(), stream.cuda_stream)
    stream.synchronize()
    s = {"kind": "decode", "size": (bx, by, w, h), "blocks": blocks, "error": c["error"], "stream": stream}
    if c["error"]:
        s["image"], s["out"] = img, torch.zeros(4, dtype=torch.int64, device="cuda")
    else:
        s["out"] = torch.zeros(h, w, 4, dtype=torch.uint8, device="cuda")
    return s


def _run_decode(s):
    if s["error"]:
        ab.decode_error_device(*s["size"], s["blocks"].data_ptr(), s["image"].data_ptr(), s["out"].data_ptr(),
                               s["stream"].cuda_stream)
    else:
        ab.decode_device(*s["size"], s["blocks"].data_ptr(), s["out"].data_ptr(), s["stream"].cuda_stream)
    return s["out"]


_PARAMS = ("w1", "b1", "w2", "b2", "w3", "b3")


def _train_inputs(c, seed):
    """A batch of real block texels, with labels spread like the full search's (half of the
    blocks single-partition), and its layout."""
    lay = proposal.Layout(c["bx"], c["by"])
    side = 64 * max(c["bx"], c["by"])
    texels = proposal.block_rgba8(_texture(side, side, seed).cpu().numpy(), c["bx"], c["by"])
    rng = np.random.default_rng(seed + 1)
    texels = texels[rng.permutation(len(texels))[: c["rows"]]]
    x = proposal.network_inputs(texels, lay.inputs_padded)
    part = np.where(rng.random(len(x)) < 0.5, lay.p1, rng.integers(0, lay.p1, len(x))).astype(np.int32)
    bm = rng.integers(0, lay.nbm, len(x)).astype(np.int32)
    return lay, x, part, bm


def _prepare_train(c, seed):
    lay, x, part, bm = _train_inputs(c, seed)
    trainer = proposal.Trainer(lay, _network(c["bx"], c["by"]), batch=c["rows"])
    dev = torch.device("cuda")
    return {"kind": "train", "trainer": trainer, "x": torch.from_numpy(x).to(dev), "part": torch.from_numpy(part).to(dev),
            "bm": torch.from_numpy(bm).to(dev), "rows": c["rows"]}


def _run_train(s):
    t = s["trainer"]
    with torch.cuda.stream(t.stream):
        t.forward(s["x"], s["rows"])
        loss = t.backward(s["x"], s["part"], s["bm"], s["rows"])
    return {"logits": t.z, "loss": loss, "grads": {k: t.g[k] for k in _PARAMS}}


_PREPARE = {"encode": _prepare_encode, "batch": _prepare_batch, "mipchain": _prepare_mipchain, "decode": _prepare_decode,
            "train": _prepare_train}
_RUN = {"encode": _run_encode, "batch": _run_batch, "mipchain": _run_mipchain, "decode": _run_decode, "train": _run_train}


# ------------------------------------------------------------ what a pass needs

def _encode_work(w, h, bx, by, net):
    """Texels in, blocks out; the full search's operations by the op-count model of the
    reference's passes, or the proposal network's (what its search does after them depends on
    the texture)."""
    lib = ab.load_library()
    n = _blocks(w, h, bx, by)
    flops = flop_model.mlp_flops(lib, bx, by) if net else flop_model.per_block(lib, bx, by)["total"]
    return {"bytes": 4.0 * w * h + 16.0 * n, "flops": flops * n}


def work(case):
    c = case
    if c["kind"] == "encode":
        return _encode_work(c["w"], c["h"], c["bx"], c["by"], c["search"] == "proposal")
    if c["kind"] in ("batch", "mipchain"):
        if c["kind"] == "batch":
            parts = [_encode_work(w, h, bx, by, False) for w, h, bx, by in _batch_sizes(c)]
        else:
            parts = [_encode_work(w, h, c["bx"], c["by"], True) for w, h in ab.mip_dims(c["w"], c["h"])]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if c["kind"] == "decode":
        return {"bytes": 4.0 * c["w"] * c["h"] + 16.0 * _blocks(c["w"], c["h"], c["bx"], c["by"]), "flops": 0.0}
    lay = proposal.Layout(c["bx"], c["by"])
    hid, n = proposal.HIDDEN, c["rows"]
    params = hid * (lay.inputs_padded + 1) + hid * (hid + 1) + lay.outputs * (hid + 1)
    macs = n * (lay.inputs_padded * hid + hid * hid + hid * lay.outputs)
    # inputs, labels, weights and gradients, logits and losses; three products of each layer
    # but the first layer's input gradient
    return {"bytes": 4.0 * (n * (lay.inputs_padded + 4 + lay.outputs) + 2 * params),
            "flops": 2.0 * (3 * macs - n * lay.inputs_padded * hid)}


def exact(case, seed):
    """The training step in 64 bits; every other output is bytes or whole numbers."""
    if case["kind"] != "train":
        return None
    lay, x, part, bm = _train_inputs(case, seed)
    net = dict(_network(case["bx"], case["by"]))
    w1 = np.zeros((proposal.HIDDEN, lay.inputs_padded), np.float32)
    w1[:, : lay.inputs] = net["w1"]
    net["w1"] = w1
    dev = torch.device("cuda")
    p = {k: torch.from_numpy(np.ascontiguousarray(net[k])).to(dev).double().requires_grad_() for k in _PARAMS}
    xd = torch.from_numpy(x).to(dev).double()
    rows = torch.arange(len(x), device=dev)
    pl = torch.from_numpy(part).to(dev).long()
    h = torch.relu(xd @ p["w1"].T + p["b1"])
    h = torch.relu(h @ p["w2"].T + p["b2"])
    z = h @ p["w3"].T + p["b3"]
    zp = z[:, : lay.p1 + 1]
    loss_part = torch.logsumexp(zp, 1) - zp[rows, pl]
    heads = torch.from_numpy(lay.head_of(part)).to(dev).long()
    cols = lay.head_base + heads[:, None] * lay.head_stride + torch.arange(lay.nbm, device=dev)
    zh = torch.gather(z, 1, cols)
    loss_bm = torch.logsumexp(zh, 1) - zh[rows, torch.from_numpy(bm).to(dev).long()]
    ((loss_part + loss_bm).sum() / len(x)).backward()
    return {"logits": z.detach(), "loss": torch.stack([loss_part, loss_bm], 1).detach(), "grads": {k: p[k].grad for k in _PARAMS}}

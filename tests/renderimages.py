"""Small render-temporal file images with chosen leaf kinds, for the decode tests: grid resolutions, FP16 and FP32
keys, fine grids, Mode2 shells.  Leaf layout: src/render_temporal_payload.cpp:62-107, 234-311; file layout:
render/src/vbt_file.cpp:39-206."""
import struct

import numpy as np


def _stream(rng, controls, bins, frames, codec):
    """A control stream of random keys (the first and last frame among them), and its key count."""
    desc, hints, keys, start = [], bytearray(), bytearray(), 0
    for _ in range(controls):
        f = np.unique(np.concatenate([[0, frames - 1], rng.choice(frames, rng.integers(0, 9))]))
        v = rng.normal(0, 1, len(f)).astype(np.float16)
        at = [max(0, int(np.searchsorted(f, b * frames // bins)) - 1) for b in range(bins)]
        desc.append(start | (len(f) << 16) | (1 << 24))
        hints += bytes(at)
        for t, x in zip(f, v):
            keys += struct.pack("<HHf", t, 0, float(x) * 1.01) if codec == 1 else struct.pack("<B", t) + x.tobytes()
        start += len(f)
    pad = lambda b: bytes(b) + bytes(-len(b) % 4)
    return struct.pack(f"<{controls}I", *desc) + pad(hints) + pad(keys), start


def render_image(dims, frames, kinds, seed=0):
    """File image (numpy uint8) whose leaf i is of kind kinds[i % len(kinds)]: None for an EMPTY leaf, else a dict
    of res (coarse resolution) and, optionally, fine (fine resolution) or shell (share of voxels), fp32 (FP32 keys
    in the coarse stream), fp32_second (in the other)."""
    rng = np.random.default_rng(seed)
    L = int(np.prod([-(-d // 8) for d in dims]))
    blocks = []
    for i in range(L):
        k = kinds[i % len(kinds)]
        if k is None:
            blocks.append(struct.pack("<I", 4 << 6))
            continue
        c, c2 = (1 if k.get("fp32") else 0), (1 if k.get("fp32_second") else 0)
        coarse, n1 = _stream(rng, k["res"] ** 3, 8, frames, c)
        mode, second, n2 = 1, b"", 0
        if "fine" in k:
            mode = 3
            second, n2 = _stream(rng, k["fine"] ** 3, 8, frames, c2)
        elif "shell" in k:
            mode = 2
            on = rng.random(512) < k["shell"]
            on[0] = True
            second, n2 = _stream(rng, int(on.sum()), 4, frames, c2)
            group = np.concatenate([[0], np.cumsum(on.reshape(8, 64).sum(1))[:-1]]).astype("<u2")
            second = np.packbits(on, bitorder="little").tobytes() + group.tobytes() + second
        blocks.append(struct.pack("<II", mode | (c << 2) | (c2 << 4) | (k["res"] << 6) | (k.get("fine", 0) << 9), n1 | (n2 << 16)) +
                      coarse + second)
    off = np.concatenate([[0], np.cumsum([len(b) // 4 for b in blocks])]).astype("<u4")
    return np.frombuffer(b"VBTPACK4" + struct.pack("<11I", 4, *dims, frames, 8, 4, 0, L, 1, 0) + off.tobytes() + b"".join(blocks),
                         np.uint8).copy()

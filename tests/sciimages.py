"""Small scientific (generic profile) file images with chosen leaf kinds, for the decode tests: coefficients per
control, events of every tier and order, residual grids of every width and subtype.  Leaf layout:
render/src/scientific_decode.cpp:82-359; file layout: render/src/vbt_file.cpp:39-206."""
import struct

import numpy as np

EVENT_CAPS = (64, 256, 768, 1024)


def _events(rng, frames, count, tier, fpb, spread, swap):
    """An event section: `count` events on frames [spread[0], spread[1]), in the order of their bins and keys, or
    with two neighbouring keys of a bin exchanged (swap)."""
    cap = EVENT_CAPS[tier]
    lo, hi = spread or (0, frames)
    at = np.sort(rng.choice((hi - lo) * 512, count, replace=False)) + lo * 512
    t, voxel = at // 512, at % 512
    bins = np.minimum(15, t // fpb)
    key = (((t - bins * fpb) << 9) | voxel) & 0xFFFF
    order = np.lexsort((key, bins))
    bins, key = bins[order], key[order].astype(np.uint16)
    if swap:
        i = int(np.flatnonzero(bins[1:] == bins[:-1])[0])
        key[[i, i + 1]] = key[[i + 1, i]]
    mask = np.zeros(512, np.uint8)
    mask[voxel] = 1
    start = np.searchsorted(bins, np.arange(16)).astype("<u2")
    keys = np.zeros(cap, "<u2")
    keys[:count] = key
    nib = np.zeros(cap, np.uint8)
    nib[:count] = rng.integers(0, 16, count)
    return (struct.pack("<f", rng.uniform(0.1, 0.4)) + np.packbits(mask, bitorder="little").tobytes() + start.tobytes() +
            keys.tobytes() + (nib[0::2] | (nib[1::2] << 4)).tobytes())


def _codes(rng, grids, per, bits):
    n = (per * bits + 7) // 8
    return rng.integers(0, 256, grids * n, dtype=np.uint8).tobytes()


def sci_image(dims, frames, kinds, seed=0):
    """File image (numpy uint8) whose leaf i is of kind kinds[i % len(kinds)]: a dict of keep (coefficients per
    control) and, for events: events, tier, fpb, spread, swap; for a residual grid: res (3 or 4), bits, tkeep (0:
    a grid per frame, else that many temporal-basis grids)."""
    rng = np.random.default_rng(seed)
    L = int(np.prod([-(-d // 8) for d in dims]))
    top = max(k["keep"] for k in kinds)
    scales = rng.uniform(0.002, 0.01, top - 1).astype("<f4")
    blocks = []
    for i in range(L):
        k = kinds[i % len(kinds)]
        keep = k["keep"]
        rec = np.zeros((64, keep + 1), np.uint8)
        rec[:, :2] = rng.normal(0, 1, (64, 1)).astype("<f2").view(np.uint8)
        rec[:, 2:] = rng.integers(0, 256, (64, keep - 1))
        head, body = (keep - 1) << 2, b""
        if "events" in k:
            tier, fpb = k.get("tier", 1), k.get("fpb", -(-frames // 16))
            head |= 1 | (tier << 8) | ((fpb - 1) << 10) | (k["events"] << 16)
            body = _events(rng, frames, k["events"], tier, fpb, k.get("spread"), k.get("swap", False))
        elif "res" in k:
            tkeep, per = k.get("tkeep", 0), k["res"] ** 3
            head |= (k["res"] - 1) | (k["bits"] << 8) | ((1 << 12) | ((tkeep - 1) << 15) if tkeep else 0)
            grids = tkeep or frames
            body = rng.uniform(0.05, 0.25, grids).astype("<f2").tobytes() + _codes(rng, grids, per, k["bits"])
        b = struct.pack("<I", head) + rec.tobytes() + body
        blocks.append(b + bytes(-len(b) % 4))
    off = np.concatenate([[0], np.cumsum([len(b) // 4 for b in blocks])]).astype("<u4")
    return np.frombuffer(b"VBTPACK4" + struct.pack("<11I", 4, *dims, frames, 8, 4, top, L, 2, top - 1) + scales.tobytes() +
                         off.tobytes() + b"".join(blocks), np.uint8).copy()

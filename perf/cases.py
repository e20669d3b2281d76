"""The work a user of vbt_b200 has it do, as cases that can be timed and compared.

listed() names the cases, draw() gives others of the same ranges, prepare() makes what a program has
in hand before the call (assets opened from VBTPACK4 file images, query lists, rays, output
buffers), run() is one pass through the public entry points, work() the bytes and operations a pass
cannot do without, and exact() the values a pass should give, from plain torch in 64 bits.

The files are written here from seeded fields, in plain torch: a smoke plume in a rising cone (most
leaves EMPTY), a fire that fills its volume, a liquid level set with Mode2 shell leaves, and a
scientific field with sparse events, dense residual grids and plain coarse leaves.  The control
series follow the moving fields, and a series keeps as keys its ends, every 12th frame and the
frames where it bends, which gives the files the key counts and sizes of encoded ones (about a third
of the frames; 10 to 20 KB for a render leaf, 1 KB for a scientific one).
"""
import math
import struct

import numpy as np
import torch

import vbt_b200 as vbt
from vbt_b200.encode import encode_render_temporal

DEV = "cuda:0"
KEY_SHARE = 0.4           # keys per control and frame, about
FINE_SHARE = 0.4          # FINE6 leaves of a density file, the others are GRID4
KEEP = 4                  # temporal coefficients of a scientific control
CHUNK = 1 << 23


# ------------------------------------------------------------------------------------- the cases
def listed():
    def case(name, kind, asset, x, y, z, t, n, **kw):
        return dict(name=name, kind=kind, asset=asset, x=x, y=y, z=z, t=t, n=n, **kw)
    return [
        # a probe of a few voxels in a small volume: launch and latency only
        case("points_small", "points", "fire", 64, 64, 64, 24, 1000),
        # a simulation or analysis step that reads a million random space-time points of a plume
        case("points_smoke", "points", "smoke", 256, 256, 256, 96, 1_000_000),
        # the same of a scientific field
        case("points_sci", "points", "sci", 128, 128, 128, 64, 1_000_000),
        # a viewer's z-slice over a range of time
        case("slice_fire", "slice", "fire", 128, 128, 192, 40, 16),
        # playback: the page table and the voxel cache of the frame shown now, a volume whose sides are not
        # multiples of the leaf's
        case("frame_fire", "frame", "fire", 125, 131, 190, 40, 1),
        # a whole timeline of a sparse plume into a ring of caches, tuned and captured once
        case("timeline_smoke", "timeline", "smoke", 256, 256, 256, 96, 96),
        # dense frames of a liquid for a tool that wants plain volumes
        case("dense_levelset", "dense", "levelset", 192, 160, 176, 40, 32),
        # all frames of a scientific field, exact
        case("dense_sci", "dense", "sci", 128, 128, 128, 64, 64),
        # the same window of time by the tensor cores
        case("window_sci", "window", "sci", 128, 128, 128, 64, 64),
        # one rendered view of a fire: the frame's control cache and a density sum along each pixel's ray
        case("rays_fire", "rays", "fire", 128, 128, 192, 40, 1280 * 720),
        # encoding a simulated density field
        case("encode_density", "encode", "blobs", 100, 88, 96, 40, 40),
        # the serving loop: point batches, slices and frames over four resident files
        case("serve_mix", "serve", "mix", 128, 112, 120, 48, 40),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["points", "points", "slice", "frame", "timeline", "dense", "dense", "window", "rays", "encode",
                       "serve"])
    side = lambda lo, hi: _log_int(rng, lo, hi)  # noqa: E731
    if kind == "encode":
        t = rng.randint(9, 40)
        return dict(kind=kind, asset="blobs", x=side(24, 96), y=side(24, 88), z=side(24, 96), t=t, n=t)
    if kind == "serve":
        return dict(kind=kind, asset="mix", x=side(48, 120), y=side(48, 112), z=side(48, 112), t=rng.randint(12, 48),
                    n=rng.randint(4, 40))
    asset = rng.choice(["smoke", "fire", "levelset", "sci"])
    if kind == "window":
        asset = rng.choice(["fire", "sci"])
    elif kind == "rays":
        asset = rng.choice(["smoke", "fire"])
    top = {"smoke": 200, "fire": 128, "levelset": 128, "sci": 128}[asset]
    x, y, z = side(40, top), side(40, top), side(40, top)
    t = rng.randint(16, 64) if asset == "sci" else rng.randint(12, 96 if asset == "smoke" else 48)
    if kind == "points":
        n = _log_int(rng, 500, 1_000_000)
    elif kind == "rays":
        n = _log_int(rng, 20_000, 900_000)
    elif kind == "frame":
        n = 1
    elif kind == "slice":
        n = rng.randint(1, min(t, 16))
    elif kind == "window":
        n = min(t, rng.choice([16, 32, 64]))
    else:
        n = min(rng.randint(min(t, 4), t), max(4, 300_000_000 // (x * y * z)))
    return dict(kind=kind, asset=asset, x=x, y=y, z=z, t=t, n=n)


def _leaves(c):
    return -(-c["x"] // 8) * (-(-c["y"] // 8)) * (-(-c["z"] // 8))


def _leaf_bytes(asset, t):
    if asset == "sci":
        return 4 + 64 * (KEEP + 1) + 740
    keys = KEY_SHARE * t
    if asset == "levelset":
        return 8 + 64 * (12 + 3 * keys) + 0.3 * 512 * (8 + 3 * keys)
    return 8 + 64 * (12 + 3 * keys) + FINE_SHARE * 216 * (12 + 3 * keys)


def _share(asset):
    """Share of non-EMPTY leaves."""
    return 0.12 if asset == "smoke" else 1.0


def work(case):
    c = case
    kind, n, vox = c["kind"], c["n"], c["x"] * c["y"] * c["z"]
    active = _leaves(c) * _share(c["asset"])
    file = active * _leaf_bytes(c["asset"], c["t"]) if c["asset"] not in ("mix", "blobs") else 0.0
    # one frame of a leaf: descriptors, two bin bytes and two keys of each control
    once = active * (64 + FINE_SHARE * 216) * 12 if c["asset"] != "sci" else file
    if kind == "points":
        hit = n * _share(c["asset"])
        return {"bytes": 20.0 * n + hit * 8 * 12, "flops": hit * 50.0}
    if kind == "slice":
        part = 8.0 / c["z"]
        return {"bytes": 4.0 * n * c["x"] * c["y"] + min(file, once * n) * part, "flops": 10.0 * n * c["x"] * c["y"]}
    if kind == "frame":
        return {"bytes": active * 2048.0 + once + 12.0 * _leaves(c), "flops": active * 512 * 15.0}
    if kind in ("timeline", "window"):
        return {"bytes": n * active * 2048.0 + file, "flops": n * active * 512 * 15.0}
    if kind == "dense":
        return {"bytes": 4.0 * n * vox + file, "flops": n * active * 512 * 15.0}
    if kind == "rays":
        return {"bytes": 64.0 * n + once + active * 280 * 4, "flops": 256.0 * 60 * n * _share(c["asset"])}
    if kind == "encode":
        return {"bytes": 4.0 * vox * n + 0.5 * vox * n, "flops": 40.0 * vox * n}
    points = sum(r[2] for r in _requests(c, 0) if r[0] == "points")
    values = sum((r[4] - r[3]) * c["x"] * c["y"] for r in _requests(c, 0) if r[0] == "slice")
    values += sum(vox for r in _requests(c, 0) if r[0] == "frames")
    return {"bytes": 60.0 * points + 8.0 * values, "flops": 30.0 * points + 15.0 * values}


# ------------------------------------------------------------------------------------- the fields
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


class _Noise:
    """A sum of cosines with wavelengths of 10 to 80 voxels that moves and changes slowly, about 0.5."""

    def __init__(self, seed, modes=14):
        r = np.random.default_rng(seed)
        d = r.normal(size=(modes, 3))
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        wave = np.exp(r.uniform(np.log(10.0), np.log(80.0), modes))
        self.k = 2 * np.pi * d / wave[:, None]
        self.w = self.k @ np.array([0.0, 0.0, 1.0]) + r.normal(0.0, 0.05, modes)
        self.phi = r.uniform(0, 2 * np.pi, modes)
        self.a = np.sqrt(wave) / np.sqrt(wave).sum() * 1.6

    def __call__(self, x, y, z, t):
        out = torch.full_like(x, 0.5).unsqueeze(-1).expand(*x.shape, t.numel()).clone()
        for k, w, p, a in zip(self.k, self.w, self.phi, self.a):
            at = (float(k[0]) * x + float(k[1]) * y + float(k[2]) * z + float(p)).unsqueeze(-1)
            out += float(a) * torch.cos(at - float(w) * t)
        return out


class _Field:
    """Value of a scene at positions [...] and all frames: [..., frames] float32."""

    def __init__(self, asset, dims, frames, seed):
        self.asset, self.dims = asset, dims
        self.t = torch.arange(frames, device=DEV, dtype=torch.float32)
        self.noise = _Noise(seed)
        r = np.random.default_rng(seed + 77)
        X, Y, Z = dims
        self.balls = np.stack([r.uniform(0, X, 12), r.uniform(0, Y, 12), r.uniform(0.4 * Z, 0.9 * Z, 12),
                               r.uniform(-0.5, 0.5, 12), r.uniform(-0.5, 0.5, 12), r.uniform(0, 1, 12),
                               r.uniform(3, 9, 12)], 1)
        self.swing = r.uniform(0, 2 * np.pi)

    def cone(self, x, y, z):
        X, Y, Z = self.dims
        r = torch.sqrt((x - X / 2) ** 2 + (y - Y / 2) ** 2)
        return 0.06 * X + 0.34 * (z - 0.04 * Z) * X / Z - r

    def __call__(self, x, y, z):
        if self.asset == "levelset":
            Z, t = self.dims[2], self.t
            wave = 0.03 * Z * torch.sin(0.05 * x.unsqueeze(-1) + 0.1 * t + self.swing)
            phi = z.unsqueeze(-1) - (0.4 * Z + wave)
            for cx, cy, cz, vx, vy, vz, rad in self.balls:
                dx, dy = x.unsqueeze(-1) - (cx + vx * t), y.unsqueeze(-1) - (cy + vy * t)
                dz = z.unsqueeze(-1) - (cz + vz * t - 0.025 * t * t)
                phi = torch.minimum(phi, torch.sqrt(dx * dx + dy * dy + dz * dz) - rad)
            return phi
        v = self.noise(x, y, z, self.t)
        if self.asset == "sci":
            return 4.0 * (v - 0.5)
        v = torch.clamp((v - 0.3) * 2.0, 0.0, 1.0)
        if self.asset == "smoke":
            top = 0.3 * self.dims[2] + 1.5 * self.t
            v = v * torch.clamp(self.cone(x, y, z) / 6.0, 0.0, 1.0).unsqueeze(-1)
            v = v * torch.clamp((top - z.unsqueeze(-1)) / 8.0, 0.0, 1.0)
        return v


def _keys(series, eps):
    """Which frames of [..., T] are keys, and the values they are stored with (binary16)."""
    T = series.shape[-1]
    key = torch.zeros(series.shape, dtype=torch.bool, device=DEV)
    key[..., 0] = key[..., -1] = True
    key[..., ::12] = True
    if T > 2:
        key[..., 1:-1] |= (series[..., 2:] - 2 * series[..., 1:-1] + series[..., :-2]).abs() > eps
    return key, series.half()


def _between(key, val):
    """The series that keys and their values stand for, in 64 bits: linear between two keys."""
    T = key.shape[-1]
    t = torch.arange(T, device=DEV)
    at = torch.where(key, t, -1).cummax(-1).values
    nx = torch.where(key, t, T - 1).flip(-1).cummin(-1).values.flip(-1)
    v = val.double()
    v0, v1 = v.gather(-1, at), v.gather(-1, nx)
    return v0 + torch.where(nx > at, (t - at) / (nx - at).clamp(min=1), 0.0) * (v1 - v0)


def _axis(pos, res):
    """Lower control and weight of a position in a leaf on a grid of `res` controls over 0 .. 7."""
    f = pos.clamp(0, 7) * ((res - 1) / 7.0)
    i = f.floor().clamp(0, res - 2)
    return i.long(), f - i


def _mix(grid, row, lx, ly, lz, t, res):
    """Trilinear sample of grid [rows, res^3, T or 1] at leaf positions, in 64 bits."""
    (x, tx), (y, ty), (z, tz) = _axis(lx, res), _axis(ly, res), _axis(lz, res)
    out = torch.zeros(lx.shape, dtype=torch.float64, device=DEV)
    for k in range(8):
        a, b, c = k & 1, (k >> 1) & 1, k >> 2
        w = (tx if a else 1 - tx) * (ty if b else 1 - ty) * (tz if c else 1 - tz)
        out += w * grid[row, ((z + c) * res + y + b) * res + x + a, t].double()
    return out


# ------------------------------------------------------------------------------------- the files
class _File:
    """The layout shared by the kinds of files: leaf grid, header, bytes."""

    def __init__(self, asset, dims, frames, seed):
        self.asset, self.dims, self.frames = asset, dims, frames
        self.grid = tuple(-(-d // 8) for d in dims)
        self.leaves = self.grid[0] * self.grid[1] * self.grid[2]
        self.field = _Field(asset, dims, frames, seed)
        self.gen = _gen(seed)

    def corner(self, leaf):
        gx, gy, _ = self.grid
        return [(8 * v).float() for v in (leaf % gx, (leaf // gx) % gy, leaf // (gx * gy))]

    def positions(self, leaf, res):
        """World positions [leaves, res^3] of a leaf's controls (res 8: of its voxels)."""
        x, y, z = self.corner(leaf)
        i = torch.arange(res ** 3, device=DEV)
        step = 7.0 / (res - 1)
        return (x[:, None] + (i % res) * step, y[:, None] + (i // res % res) * step, z[:, None] + (i // res ** 2) * step)

    def rand(self, *shape):
        return torch.rand(shape, generator=self.gen, device=DEV)

    def image(self, words, header, scales, put):
        """The file's bytes: leaf blocks of `words` words, filled in by put(int32 words, first word of each)."""
        off = torch.zeros(self.leaves + 1, dtype=torch.int64, device=DEV)
        off[1:] = words.cumsum(0)
        pay = torch.zeros(int(off[-1]), dtype=torch.int32, device=DEV)
        put(pay, off[:-1])
        head = b"VBTPACK4" + struct.pack("<11I", 4, *self.dims, self.frames, 8, 4, *header) + scales
        head = torch.frombuffer(bytearray(head), dtype=torch.uint8)
        return torch.cat([head, off.int().cpu().view(torch.uint8), pay.cpu().view(torch.uint8)])

    def locate(self, x, y, z):
        gx, gy, _ = self.grid
        bx, by, bz = (torch.div(v.floor().long(), 8, rounding_mode="floor") for v in (x, y, z))
        return (bz * gy + by) * gx + bx, x - 8 * bx, y - 8 * by, z - 8 * bz


def _put_bytes(pay, at, values):
    pay.view(torch.uint8)[at] = values.to(torch.uint8)


class _Stream:
    """Keyed control series [rows, C, T] as the bytes of a control stream with `bins` time bins."""

    def __init__(self, series, bins, eps, used=None):
        self.key, self.val = _keys(series, eps)
        if used is not None:
            self.key &= used.unsqueeze(-1)
        self.used, self.bins = used, bins
        self.rows, self.C, self.T = series.shape
        self.count = self.key.sum(-1)
        self.keys = self.count.sum(-1)
        self.start = self.count.cumsum(-1) - self.count
        self.controls = torch.full((self.rows,), self.C, device=DEV) if used is None else used.sum(-1)

    def words(self):
        return self.controls * (1 + self.bins // 4) + (3 * self.keys + 3) // 4

    def put(self, pay, at):
        """At word at[row]: descriptors, time bins, 3-byte keys."""
        less = torch.zeros(self.rows, self.C, self.T + 1, dtype=torch.int32, device=DEV)
        less[..., 1:] = self.key.cumsum(-1)
        first = [b * self.T // self.bins for b in range(self.bins)]
        n = less[..., first]
        hint = torch.where(n < self.count.unsqueeze(-1), n - 1, self.count.unsqueeze(-1).int() - 1).clamp(min=0)
        span = torch.cat([hint[..., 1:], self.count.unsqueeze(-1).int()], -1) - hint
        desc = self.start | (self.count << 16) | (span.amax(-1).long().clamp(1, 255) << 24)
        desc = torch.where(desc >= 1 << 31, desc - (1 << 32), desc).int()
        row_bytes = hint.to(torch.uint8).view(torch.int32)
        if self.used is None:
            place = torch.arange(self.C, device=DEV).expand(self.rows, self.C)
            sel = torch.ones(self.rows, self.C, dtype=torch.bool, device=DEV)
        else:
            place, sel = self.used.cumsum(-1) - 1, self.used
        pay[(at[:, None] + place)[sel]] = desc[sel]
        bins_at = (at + self.controls)[:, None] + place * (self.bins // 4)
        for k in range(self.bins // 4):
            pay[(bins_at + k)[sel]] = row_bytes[..., k][sel]
        pool = 4 * (at + self.controls * (1 + self.bins // 4))
        for r0 in range(0, self.rows, 2048):
            r1 = min(self.rows, r0 + 2048)
            r, c, t = self.key[r0:r1].nonzero(as_tuple=True)
            i = self.start[r0:r1][r, c] + less[r0:r1][r, c, t]
            b = pool[r0:r1][r] + 3 * i
            h = self.val[r0:r1][r, c, t].view(torch.int16)
            _put_bytes(pay, b, t)
            _put_bytes(pay, b + 1, h & 0xFF)
            _put_bytes(pay, b + 2, (h >> 8) & 0xFF)


class _RenderFile(_File):
    """A render-temporal file: GRID4 and FINE6 leaves, or GRID4 and Mode2 shell leaves of a level set."""

    def __init__(self, asset, dims, frames, seed):
        super().__init__(asset, dims, frames, seed)
        leaf = torch.arange(self.leaves, device=DEV)
        if asset == "smoke":
            x, y, z = self.corner(leaf)
            keep = (self.field.cone(x + 3.5, y + 3.5, z + 3.5) > -4.0) & (z + 8 > 0.04 * dims[2])
            keep &= z < 0.3 * dims[2] + 1.5 * frames
            leaf = leaf[keep]
        self.active = leaf
        self.rank = torch.full((self.leaves,), -1, dtype=torch.int64, device=DEV)
        self.rank[leaf] = torch.arange(leaf.numel(), device=DEV)
        level = asset == "levelset"
        self.level = level
        eps = 0.006 if asset == "smoke" else 0.02
        coarse = self.field(*self.positions(leaf, 4))
        self.coarse = _Stream(coarse, 8, eps)
        if level:
            # the voxels within three voxels of the surface at some frame, and their residual there
            box = []
            for r0 in range(0, leaf.numel(), 1024):
                part = leaf[r0:r0 + 1024]
                phi = self.field(*self.positions(part, 8))
                near = phi.abs().amin(-1) <= 3.0
                has = near.any(-1).nonzero().squeeze(-1)
                base = _between(self.coarse.key[r0:r0 + 1024][has], self.coarse.val[r0:r0 + 1024][has])
                v = torch.arange(512, device=DEV)
                t = torch.arange(frames, device=DEV)
                lx, ly, lz = ((q.double())[None, :, None] for q in (v % 8, v // 8 % 8, v // 64))
                row = torch.arange(has.numel(), device=DEV)[:, None, None]
                shape = (has.numel(), 512, frames)
                at = [q.expand(shape) for q in (lx, ly, lz)]
                low = _mix(base, row.expand(shape), *at, t.expand(shape), 4)
                box.append((r0 + has, near[has], (phi[has] - low.float())))
            self.second = torch.cat([b[0] for b in box])
            self.near = torch.cat([b[1] for b in box])
            self.extra = _Stream(torch.cat([b[2] for b in box]), 4, 0.02, self.near)
        else:
            self.second = (self.rand(leaf.numel()) < FINE_SHARE).nonzero().squeeze(-1)
            pos = self.positions(leaf[self.second], 6)
            fine = self.field(*pos) * 0.25 * torch.cos(0.9 * (pos[0] + pos[1] + pos[2])).unsqueeze(-1)
            self.extra = _Stream(fine, 8, 0.2 * eps)
        self.place = torch.full((leaf.numel(),), -1, dtype=torch.int64, device=DEV)
        self.place[self.second] = torch.arange(self.second.numel(), device=DEV)

    def bytes(self):
        A = self.active.numel()
        c_words = self.coarse.words()
        words = torch.ones(self.leaves, dtype=torch.int64, device=DEV)
        mine = 2 + c_words
        mine[self.second] += self.extra.words() + (20 if self.level else 0)
        words[self.active] = mine

        def put(pay, off):
            pay[off] = 4 << 6
            at = off[self.active]
            mode = torch.full((A,), 1 | (4 << 6), dtype=torch.int32, device=DEV)
            mode[self.second] = 2 | (4 << 6) if self.level else 3 | (4 << 6) | (6 << 9)
            pay[at] = mode
            kf = torch.zeros(A, dtype=torch.int64, device=DEV)
            kf[self.second] = self.extra.keys << 16
            kf |= self.coarse.keys
            pay[at + 1] = torch.where(kf >= 1 << 31, kf - (1 << 32), kf).int()
            self.coarse.put(pay, at + 2)
            ex = (at + 2 + c_words)[self.second]
            if self.level:
                bit = self.near.view(-1, 64, 8).to(torch.int32)
                mask = (bit << torch.arange(8, device=DEV, dtype=torch.int32)).sum(-1)
                group = self.near.view(-1, 8, 64).sum(-1)
                before = group.cumsum(-1) - group
                both = torch.stack([before & 0xFF, before >> 8], -1).view(-1, 16)
                rows = torch.cat([mask, both], 1)
                _put_bytes(pay, 4 * ex[:, None] + torch.arange(80, device=DEV), rows)
                ex = ex + 20
            self.extra.put(pay, ex)
        return self.image(words, (0, self.leaves, 1, 0), b"", put)

    def solve(self):
        self.c64 = _between(self.coarse.key, self.coarse.val)
        key = self.extra.key.clone()
        key[..., 0] = True          # unused voxels of a shell: any series will do
        self.x64 = _between(key, self.extra.val)
        return self

    def value(self, x, y, z, t):
        leaf, lx, ly, lz = self.locate(x, y, z)
        rank = self.rank[leaf]
        out = torch.zeros(x.shape, dtype=torch.float64, device=DEV)
        on = (rank >= 0).nonzero().squeeze(-1)
        rank, lx, ly, lz, t = rank[on], lx[on], ly[on], lz[on], t[on]
        v = _mix(self.c64, rank, lx, ly, lz, t, 4)
        two = (self.place[rank] >= 0).nonzero().squeeze(-1)
        row, ax, ay, az = self.place[rank[two]], lx[two], ly[two], lz[two]
        if self.level:
            vox = ((az * 8 + ay) * 8 + ax).long()
            near = self.near[row, vox]
            v2 = v[two] + torch.where(near, self.x64[row, vox, t[two]], 0.0)
            v[two] = torch.where(near, v2, v2.clamp(min=0.0))
        else:
            v[two] += _mix(self.x64, row, ax, ay, az, t[two], 6)
        out[on] = v
        return out


class _SciFile(_File):
    """A scientific file: three in five leaves with sparse events, the others plain coarse leaves or with a
    4^3 residual grid per frame."""

    def __init__(self, asset, dims, frames, seed):
        super().__init__(asset, dims, frames, seed)
        L, T = self.leaves, frames
        leaf = torch.arange(L, device=DEV)
        t = torch.arange(T, device=DEV, dtype=torch.float64)
        k = torch.arange(KEEP, device=DEV, dtype=torch.float64)
        self.basis = torch.cos(math.pi / T * (t[:, None] + 0.5) * k) * math.sqrt(2.0 / T)
        self.basis[:, 0] = math.sqrt(1.0 / T)
        coef = torch.empty(L, 64, KEEP, device=DEV)
        for r0 in range(0, L, 2048):
            coef[r0:r0 + 2048] = self.field(*self.positions(leaf[r0:r0 + 2048], 4)) @ self.basis.float()
        self.dc = coef[..., 0].half()
        self.scale = coef[..., 1:].abs().amax((0, 1)).clamp(min=1e-3) / 127.0
        self.ac = (coef[..., 1:] / self.scale).round().clamp(-127, 127).to(torch.int8)
        u = self.rand(L)
        self.mode = torch.where(u < 0.6, 1, torch.where(u < 0.8, 0, 3))
        # events: `count` increasing places in frame-major order of the leaf
        self.count = (64 + self.rand(L) * 190).long()
        j = torch.arange(256, device=DEV)
        at = ((j + 0.98 * self.rand(L, 256)) * (512.0 * T) / self.count[:, None]).long().clamp(max=512 * T - 1)
        self.has = (j < self.count[:, None]) & (self.mode == 1)[:, None]
        self.at = torch.where(self.has, at, 512 * T - 1)
        self.q = (self.rand(L, 256) * 16).long() - 8
        self.event = (1.0 + self.rand(L)) * 0.25
        self.per = -(-T // 16)
        # residual grids: 4 bits a control, a scale a frame
        self.dense = (self.mode == 3).nonzero().squeeze(-1)
        self.code = (self.rand(self.dense.numel(), T, 64) * 16).long()
        self.fs = (self.rand(self.dense.numel(), T) * 0.2 + 0.05).half()

    def bytes(self):
        L, T = self.leaves, self.frames
        rec = 64 * (KEEP + 1)
        size = torch.full((L,), 4 + rec, device=DEV)
        size += torch.where(self.mode == 1, 100 + 512 + 128, torch.where(self.mode == 3, T * 34, 0))

        def put(pay, off):
            head = self.mode | ((KEEP - 1) << 2)
            head = torch.where(self.mode == 1, head | (1 << 8) | ((self.per - 1) << 10) | (self.count << 16), head)
            head = torch.where(self.mode == 3, head | (4 << 8), head)
            pay[off] = head.int()
            body = 4 * off + 4
            h = self.dc.view(torch.int16)
            rows = torch.cat([torch.stack([h & 0xFF, (h >> 8) & 0xFF], -1), self.ac.to(torch.int16)], -1) & 0xFF
            _put_bytes(pay, body[:, None] + torch.arange(rec, device=DEV), rows.reshape(L, rec))
            one = (self.mode == 1).nonzero().squeeze(-1)
            sb = (body + rec)[one]
            pay[sb // 4] = self.event[one].view(torch.int32)
            mask = torch.zeros(one.numel(), 512, dtype=torch.bool, device=DEV)
            mask.scatter_(1, torch.where(self.has, self.at % 512, self.at[:, :1] % 512)[one], True)
            bits = (mask.view(-1, 64, 8).to(torch.int32) << torch.arange(8, device=DEV, dtype=torch.int32)).sum(-1)
            _put_bytes(pay, sb[:, None] + 4 + torch.arange(64, device=DEV), bits)
            bin_of = torch.where(self.has, self.at // 512 // self.per, 99)[one]
            start = torch.stack([(bin_of < b).sum(-1) for b in range(16)], -1)
            both = torch.stack([start & 0xFF, start >> 8], -1).view(-1, 32)
            _put_bytes(pay, sb[:, None] + 68 + torch.arange(32, device=DEV), both)
            key = torch.where(self.has, ((self.at // 512 % self.per) << 9) | (self.at % 512), 0)[one]
            both = torch.stack([key & 0xFF, key >> 8], -1).view(-1, 512)
            _put_bytes(pay, sb[:, None] + 100 + torch.arange(512, device=DEV), both)
            nib = torch.where(self.has, self.q & 15, 0)[one].view(-1, 128, 2)
            _put_bytes(pay, sb[:, None] + 612 + torch.arange(128, device=DEV), nib[..., 0] | (nib[..., 1] << 4))
            db = (body + rec)[self.dense]
            s = self.fs.view(torch.int16)
            both = torch.stack([s & 0xFF, (s >> 8) & 0xFF], -1).view(-1, 2 * T)
            _put_bytes(pay, db[:, None] + torch.arange(2 * T, device=DEV), both)
            two = self.code.view(-1, T * 32, 2)
            _put_bytes(pay, db[:, None] + 2 * T + torch.arange(32 * T, device=DEV), two[..., 0] | (two[..., 1] << 4))
        scales = self.scale.cpu().numpy().astype("<f4").tobytes()
        return self.image((size + 3) // 4, (KEEP, L, 2, KEEP - 1), scales, put)

    def solve(self):
        coef = torch.cat([self.dc.double().unsqueeze(-1), self.ac.double() * self.scale.double()], -1)
        self.c64 = coef @ self.basis.T
        norm = (self.code.double() / 15.0 * 2.0 - 1.0) * self.fs.double().unsqueeze(-1)
        self.g64 = norm.transpose(1, 2).contiguous()
        self.row = torch.zeros(self.leaves, dtype=torch.int64, device=DEV)
        self.row[self.dense] = torch.arange(self.dense.numel(), device=DEV)
        # the events of all leaves, by place
        span = 512 * self.frames
        hit = self.has.nonzero(as_tuple=True)
        self.where = hit[0] * span + self.at[hit]
        self.what = self.q[hit].double() * self.event.double()[hit[0]]
        return self

    def value(self, x, y, z, t):
        leaf, lx, ly, lz = self.locate(x, y, z)
        v = _mix(self.c64, leaf, lx, ly, lz, t, 4)
        place = leaf * (512 * self.frames) + t * 512 + ((lz * 8 + ly) * 8 + lx).long()
        i = torch.searchsorted(self.where, place).clamp(max=max(0, self.where.numel() - 1))
        if self.where.numel():
            v += torch.where(self.where[i] == place, self.what[i], 0.0)
        d = (self.mode[leaf] == 3).nonzero().squeeze(-1)
        if d.numel():
            v[d] += _mix(self.g64, self.row[leaf[d]], lx[d], ly[d], lz[d], t[d], 4)
        return v


def _file(asset, dims, frames, seed):
    return (_SciFile if asset == "sci" else _RenderFile)(asset, dims, frames, seed)


def _dims(c):
    return c["x"], c["y"], c["z"]


# ------------------------------------------------------------------------------- inputs of the calls
def _queries(dims, frames, n, seed):
    g = _gen(seed + 5)
    top = torch.tensor([*dims, frames], device=DEV)
    return (torch.rand(n, 4, generator=g, device=DEV, dtype=torch.float64) * top).int()


def _rays(dims, n, seed):
    """A pinhole view of the volume from outside: rays that start and end where they cross its box."""
    r = np.random.default_rng(seed + 6)
    h = max(1, int(math.sqrt(n * 9 / 16)))
    w = n // h
    box = torch.tensor(dims, device=DEV, dtype=torch.float64)
    turn = r.uniform(0, 2 * math.pi)
    eye = box / 2 + torch.tensor([math.cos(turn), math.sin(turn), 0.35], device=DEV, dtype=torch.float64) * 1.5 * box.max()
    fwd = torch.nn.functional.normalize(box / 2 - eye, dim=0)
    up = torch.tensor([0.0, 0.0, 1.0], device=DEV, dtype=torch.float64)
    right = torch.nn.functional.normalize(torch.linalg.cross(fwd, up), dim=0)
    down = torch.linalg.cross(fwd, right)
    i = torch.arange(n, device=DEV)
    u = ((i % w).double() + 0.5) / w - 0.5
    v = ((i // w).double() + 0.5) / h - 0.5
    d = torch.nn.functional.normalize(fwd + 0.75 * u[:, None] * right + 0.75 * h / w * v[:, None] * down, dim=1)
    a, b = (0.0 - eye) / d, (box - 1.0 - eye) / d
    near, far = torch.minimum(a, b).amax(1).clamp(min=0), torch.maximum(a, b).amin(1)
    hit = far > near
    rays = torch.zeros(n, 8, device=DEV)
    rays[:, 0:3] = (eye + d * torch.where(hit, near, 0.0)[:, None]).float()
    rays[:, 4:7] = d.float()
    rays[:, 7] = torch.where(hit, far - near, 0.0).float()
    return rays


STEPS = 256
MIX = ("smoke", "fire", "levelset", "sci")


def _requests(c, seed):
    """The requests of a serving step: 70% point batches, 20% slices over up to 16 frames, 10% frames."""
    r = np.random.default_rng(seed + 11)
    out = []
    for i in range(c["n"]):
        a = int(r.integers(len(MIX)))
        u = (i * 0.618034) % 1.0
        if u < 0.7:
            out.append(("points", a, int(10 ** (3.0 + 2.3 * ((i * 0.754878) % 1.0))), int(r.integers(1 << 30))))
        elif u < 0.9:
            n = 1 + int(15 * ((i * 0.569840) % 1.0))
            t0 = int(r.integers(0, max(1, c["t"] - n + 1)))
            out.append(("slice", a, int(r.integers(0, c["z"])), t0, min(c["t"], t0 + n)))
        else:
            out.append(("frames", a, int(r.integers(0, c["t"]))))
    return out


def _size(c, req):
    if req[0] == "points":
        return req[2]
    return (req[4] - req[3]) * c["x"] * c["y"] if req[0] == "slice" else c["x"] * c["y"] * c["z"]


def _blobs(c, seed):
    """A sum of six Gaussian blobs on straight paths plus a little noise, frame-major."""
    X, Y, Z = _dims(c)
    g, r = _gen(seed), np.random.default_rng(seed)
    out = torch.empty(c["t"], Z, Y, X, device=DEV)
    x, y, z = (torch.arange(n, device=DEV, dtype=torch.float32) for n in (X, Y, Z))
    at, go = r.uniform(0.2, 0.8, (6, 3)) * np.array([X, Y, Z]), r.uniform(-0.57, 0.57, (6, 3))
    sig, amp = r.uniform(4, 10, 6), r.uniform(0.2, 1.0, 6)
    for t in range(c["t"]):
        f = torch.randn(Z, Y, X, generator=g, device=DEV) * 0.01
        for b in range(6):
            e = [torch.exp(-(q - float(at[b, k] + go[b, k] * t)) ** 2 / (2 * float(sig[b]) ** 2)) for k, q in
                 enumerate((x, y, z))]
            f += float(amp[b]) * e[2][:, None, None] * e[1][None, :, None] * e[0][None, None, :]
        out[t] = f
    return out.view(c["t"], -1)


def _start(c, seed):
    """First frame of the range a call takes."""
    return int(np.random.default_rng(seed + 3).integers(0, c["t"] - c["n"] + 1)) if c["n"] < c["t"] else 0


def _z(c, seed):
    return int(np.random.default_rng(seed + 4).integers(0, c["z"]))


# ------------------------------------------------------------------------------------- the passes
def prepare(case, seed):
    c = case
    kind, dims, T, n = c["kind"], _dims(c), c["t"], c["n"]
    if kind == "encode":
        # the file is put together in a buffer that holds any payload of this size
        room = _leaves(c) * (24 + 280 * (3 + 3 * (T + 1) // 4))
        return {"kind": kind, "field": _blobs(c, seed), "dims": dims,
                "file": torch.zeros(room, dtype=torch.int32, device=DEV)}
    if kind == "serve":
        files = [vbt.Asset(data=_file(a, dims, T, seed + i).bytes()) for i, a in enumerate(MIX)]
        server = vbt.Server(hbm_budget_bytes=1 << 30, slots=4)
        s = {"server": server, "kind": kind, "ids": [server.add_asset(a) for a in files], "files": files}
        reqs = _requests(c, seed)
        s["out"] = torch.empty(sum(_size(c, r) for r in reqs), pin_memory=True)
        s["do"], at = [], 0
        for r in reqs:
            out = s["out"][at:at + _size(c, r)]
            at += out.numel()
            if r[0] == "points":
                q = _queries(dims, T, r[2], r[3]).cpu().pin_memory()
                s["do"].append(("points", r[1], q, out))
            else:
                s["do"].append((r[0], r[1], r[2:], out))
        return s
    a = vbt.Asset(data=_file(c["asset"], dims, T, seed).bytes())
    a.build_page_table()
    s = {"kind": kind, "asset": a, "t0": _start(c, seed) if kind in ("slice", "frame", "timeline", "dense", "window") else T // 2,
         "n": n}
    act = a.active_count
    if kind == "points":
        s["q"] = _queries(dims, T, n, seed)
        s["out"] = torch.empty(n, device=DEV)
    elif kind == "slice":
        s["z"] = _z(c, seed)
        s["out"] = torch.empty(n, dims[1], dims[0], device=DEV)
    elif kind == "dense":
        s["out"] = torch.empty(n, dims[2], dims[1], dims[0], device=DEV)
    elif kind == "rays":
        p = vbt.SampleParams()
        p.step_count, p.frame_index, p.voxel_size = STEPS, s["t0"], 1.0
        s["params"], s["rays"] = p, _rays(dims, n, seed)
        s["controls"] = torch.empty(1, act, 576, device=DEV)
        s["out"] = torch.empty(n, 8, device=DEV)
    else:
        s["out"] = torch.empty(n, act, 512, device=DEV)
        if kind == "timeline":
            s["stream"] = torch.cuda.Stream()
            s["stream"].wait_stream(torch.cuda.current_stream())
            a.autotune(n, s["out"], stream=s["stream"])
    return s


def run(state):
    s = state
    kind = s["kind"]
    if kind == "encode":
        _, offsets, payload = encode_render_temporal(s["field"], s["dims"])
        s["file"][:payload.numel()] = payload
        return {"offsets": offsets, "payload": s["file"]}
    if kind == "serve":
        server, tickets = s["server"], []
        for what, a, arg, out in s["do"]:
            if what == "points":
                tickets.append(server.submit_points(s["ids"][a], arg, out))
            elif what == "slice":
                tickets.append(server.submit_slice(s["ids"][a], *arg, out))
            else:
                tickets.append(server.submit_frames(s["ids"][a], list(arg), out))
        for t in tickets:
            if server.wait(t).status:
                raise RuntimeError("a request failed")
            server.release(t)
        return s["out"]
    a, out, t0, n = s["asset"], s["out"], s["t0"], s["n"]
    if kind == "points":
        a.query_points(s["q"], out)
    elif kind == "slice":
        a.query_slice(s["z"], t0, t0 + n, out)
    elif kind == "frame":
        a.build_page_table()
        a.decode_cache([t0], out)
    elif kind == "timeline":
        a.decode_cache_timeline(t0, n, out, stream=s["stream"])
    elif kind == "dense":
        a.decode_frames(list(range(t0, t0 + n)), out)
    elif kind == "window":
        a.decode_window(t0, n, out, frame_stride=out.stride(0))
    else:
        a.decode_control_cache([t0], s["controls"])
        a.sample_rays(s["controls"], s["params"], s["rays"], out)
        return {"controls": s["controls"], "rays": out}
    return out


# ------------------------------------------------------------------------------- the values in 64 bits
def _many(f, n, place):
    """f's values at the n places place(i) gives as (x, y, z, t), chunk by chunk."""
    out = torch.empty(n, dtype=torch.float64, device=DEV)
    for i0 in range(0, n, CHUNK):
        i = torch.arange(i0, min(n, i0 + CHUNK), device=DEV)
        x, y, z, t = place(i)
        out[i0:i0 + i.numel()] = f.value(x.double(), y.double(), z.double(), t)
    return out


def _box(f, dims, t0, n, z=None):
    """Dense frames [t0, t0 + n), or one z-layer of them."""
    X, Y = dims[0], dims[1]
    per = X * Y * (dims[2] if z is None else 1)

    def place(i):
        v = i % per
        return v % X, v // X % Y, v // (X * Y) if z is None else torch.full_like(v, z), t0 + i // per
    return _many(f, n * per, place)


def exact(case, seed):
    c = case
    kind, dims, T, n = c["kind"], _dims(c), c["t"], c["n"]
    if kind == "encode":
        return None
    if kind == "serve":
        files = [_file(a, dims, T, seed + i).solve() for i, a in enumerate(MIX)]
        parts = []
        for r in _requests(c, seed):
            f = files[r[1]]
            if r[0] == "points":
                q = _queries(dims, T, r[2], r[3]).long()
                parts.append(f.value(q[:, 0].double(), q[:, 1].double(), q[:, 2].double(), q[:, 3]))
            elif r[0] == "slice":
                parts.append(_box(f, dims, r[3], r[4] - r[3], r[2]))
            else:
                parts.append(_box(f, dims, r[2], 1))
        return torch.cat(parts)
    f = _file(c["asset"], dims, T, seed).solve()
    t0 = _start(c, seed)
    if kind == "points":
        q = _queries(dims, T, n, seed).long()
        return _many(f, n, lambda i: (q[i, 0], q[i, 1], q[i, 2], q[i, 3]))
    if kind == "slice":
        return _box(f, dims, t0, n, _z(c, seed)).view(n, dims[1], dims[0])
    if kind == "dense":
        return _box(f, dims, t0, n).view(n, *dims[::-1])
    if kind == "rays":
        return _exact_rays(f, dims, n, seed, T // 2)
    leaf = torch.arange(f.leaves, device=DEV) if c["asset"] == "sci" else f.active
    x, y, z = (v.long() for v in f.positions(leaf, 8))
    per = leaf.numel() * 512
    x, y, z = x.reshape(-1), y.reshape(-1), z.reshape(-1)
    inside = (x < dims[0]) & (y < dims[1]) & (z < dims[2])
    out = torch.zeros(n, per, dtype=torch.float64, device=DEV)
    at = inside.nonzero().squeeze(-1)
    for k in range(n):
        out[k, at] = _many(f, at.numel(), lambda i: (x[at[i]], y[at[i]], z[at[i]], torch.full_like(i, t0 + k)))
    return out.view(n, leaf.numel(), 512)


def _exact_rays(f, dims, n, seed, frame):
    rays = _rays(dims, n, seed).double()
    total = torch.zeros(n, 8, dtype=torch.float64, device=DEV)
    box = torch.tensor(dims, device=DEV)
    for i0 in range(0, n, 1 << 18):
        o, d, end = rays[i0:i0 + (1 << 18), 0:3], rays[i0:i0 + (1 << 18), 4:7], rays[i0:i0 + (1 << 18), 7]
        for k in range(STEPS):
            p = o + d * ((k + 0.5) / STEPS * end)[:, None]
            ok = ((p >= 0) & (p <= box - 1)).all(1).nonzero().squeeze(-1)
            p = p[ok]
            total[i0 + ok, 0] += f.value(p[:, 0], p[:, 1], p[:, 2], torch.full_like(ok, frame))
    controls = torch.zeros(1, f.active.numel(), 576, dtype=torch.float64, device=DEV)
    controls[0, :, :64] = f.c64[..., frame]
    controls[0, f.second, 64:280] = f.x64[..., frame]
    return {"controls": controls, "rays": total}

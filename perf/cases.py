"""What the speed of this framework is measured on.

Every case is a conversion as a program makes it through the C ABI
(include/pcgpu.h, reached with the ctypes mirror of the package): one file
image or several in host memory, records that already lie in device memory,
a LAZ file, a cloud converted in parts, or a queue of jobs. A pass returns
octree.bin, hierarchy.bin and metadata.json whole, as bytes in the buffers
the library hands out (a caller frees them with pcg_result_free: here when
the arrays go). All outputs are bytes, so there is nothing to compare with
64-bit arithmetic.

The clouds are the repository's synthetic workloads (terrain, hot-spots,
lattice, aerial strips, tiles); the LAZ files hold scan lines with several
returns per pulse, coded here point by point as LASzip's chunked point-wise
format wants it.
"""

import ctypes
import math
import struct

import numpy as np
import torch

import potreeconverter_b200 as pc
from potreeconverter_b200 import synth, synth_gpu

REC_LEN = {0: 20, 1: 28, 2: 26, 3: 34}
HOTSPOT_REC = 38  # point format 3 with one float32 of extra bytes
FILTER = "rgb,classification,intensity"


def listed():
    return [
        # a test plot or one object: the smallest call, launches and host work count
        dict(name="terrain_3k", kind="convert", cloud="terrain", points=3_000, extent=500.0, pdrf=2, method="poisson", source="host"),
        # one small tile read from a file into ordinary memory, averaged colours
        dict(name="terrain_200k_average", kind="convert", cloud="terrain", points=200_003, extent=300.0, pdrf=3, method="poisson_average",
             source="host"),
        # the reference's everyday job: a 2M-point file read into ordinary memory
        dict(name="terrain_2m", kind="convert", cloud="terrain", points=2_000_000, extent=500.0, pdrf=2, method="poisson", source="host"),
        # a larger file from page-locked memory with the cheapest sampler: copies and gathers
        dict(name="terrain_10m_random", kind="convert", cloud="terrain", points=10_000_001, extent=1500.0, pdrf=3, method="random", source="pinned"),
        # uneven density, averaged colours
        dict(name="hotspots_10m_average", kind="convert", cloud="hotspots", points=10_000_000, extent=2000.0, pdrf=3, method="poisson_average",
             source="resident"),
        # the headline workload: 50M points already on the device, octree.bin left there
        dict(name="hotspots_50m_resident", kind="convert", cloud="hotspots", points=50_000_000, extent=2000.0, pdrf=3, method="poisson",
             source="resident"),
        # the precision workload: most pairs near the spacing, many equal sort keys
        dict(name="lattice_8m_resident", kind="convert", cloud="lattice", points=8_000_000, extent=1024.0, pdrf=2, method="poisson", source="resident"),
        # a cloud larger than one part: tiles streamed in, pieces of octree.bin out
        dict(name="strips_6m_parts", kind="parts", cloud="strips", points=6_000_000, extent=20000.0, pdrf=3, method="poisson_average",
             source="pinned", group=2_000_000),
        # several files of different formats converted as one cloud, a few attributes kept
        dict(name="tiles_1m_attributes", kind="tiles", points=1_000_000, extent=400.0, method="poisson", attributes=FILTER),
        # a LAZ file as LASzip writes it by default: chunks of 50,000 points
        dict(name="laz_1m", kind="laz", points=1_000_000, chunk=50_000, pdrf=3, method="poisson"),
        # a LAZ file of many small chunks, no colours
        dict(name="laz_400k_small_chunks", kind="laz", points=400_123, chunk=5_000, pdrf=1, method="random"),
        # the request loop: jobs of very different sizes and samplers at once
        dict(name="queue_10", kind="queue", jobs=10, smallest=100_000, largest=2_000_000, extent=800.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    method = rng.choice(["poisson", "poisson", "poisson_average", "random"])
    kind = rng.choice(["convert"] * 5 + ["parts", "tiles", "laz", "laz", "queue"])
    if kind == "convert":
        source = rng.choice(["host", "pinned", "resident"])
        cloud = rng.choice(["terrain", "hotspots", "strips", "lattice"])
        most = {"host": 4_000_000, "pinned": 10_000_000, "resident": 30_000_000}[source]
        if method == "poisson_average" and source != "resident":
            most //= 10  # the result is copied out
        if cloud == "lattice":
            most = min(most, 8_000_000)
        pdrf = {"terrain": rng.choice([2, 3]), "lattice": 2}.get(cloud, 3)
        extent = {"terrain": round(rng.uniform(100.0, 2000.0), 1), "hotspots": 2000.0, "strips": 20000.0, "lattice": 1024.0}[cloud]
        return dict(kind=kind, cloud=cloud, points=_log(rng, 1_000, most), extent=extent, pdrf=pdrf, method=method, source=source)
    if kind == "parts":
        return dict(kind=kind, cloud="strips", points=_log(rng, 2_500_000, 8_000_000), extent=20000.0, pdrf=3, method=method, source="pinned",
                    group=rng.choice([1_000_000, 2_000_000]))
    if kind == "tiles":
        # averaging needs colours in the output, which the filter keeps
        return dict(kind=kind, points=_log(rng, 20_000, 1_000_000), extent=400.0, method=method, attributes=rng.choice(["", FILTER]))
    if kind == "laz":
        pdrf = rng.choice([2, 3]) if method == "poisson_average" else rng.choice([0, 1, 2, 3])
        return dict(kind=kind, points=_log(rng, 20_000, 1_000_000), chunk=_log(rng, 1_000, 50_000), pdrf=pdrf, method=method)
    return dict(kind=kind, jobs=rng.randint(4, 10), smallest=100_000, largest=_log(rng, 300_000, 2_000_000), extent=round(rng.uniform(100.0, 2000.0), 1))


# ------------------------------------------------------------------ clouds
def _write_columns(X, Y, Z, pdrf, gen, extra=False):
    """Point records as an [n, record length] byte tensor on the device, with
    the value ranges of the repository's workloads."""
    n, dev = X.numel(), X.device
    rec = torch.zeros((n, REC_LEN[pdrf] + (4 if extra else 0)), dtype=torch.uint8, device=dev)

    def put(off, v):
        b = v.contiguous().view(torch.uint8).view(n, -1)
        rec[:, off:off + b.shape[1]] = b

    def rand(lo, hi, dtype):
        return torch.randint(lo, hi, (n,), generator=gen, device=dev).to(dtype)

    for a, v in enumerate((X, Y, Z)):
        put(4 * a, v)
    put(12, rand(-32768, 32768, torch.int16))
    nret = rand(1, 6, torch.uint8)
    put(14, torch.minimum(rand(1, 6, torch.uint8), nret) | (nret << 3))
    put(15, rand(0, 32, torch.uint8))
    put(16, rand(-30, 31, torch.int8))
    put(17, rand(0, 256, torch.uint8))
    put(18, rand(0, 64, torch.int16))
    at = 20
    if pdrf in (1, 3):
        put(at, torch.arange(n, device=dev, dtype=torch.float64) * 1e-4 + 3.0e5)
        at += 8
    if pdrf in (2, 3):
        ramp = (Z - Z.min()).to(torch.float32) / max(float(Z.max() - Z.min()), 1.0)
        for k, v in enumerate((ramp, 1 - (ramp - 0.5).abs() * 2, 1 - ramp)):
            noise = torch.rand(n, generator=gen, device=dev) * 4000 + 4000
            put(at + 2 * k, (v * 50000 + noise).to(torch.int32).to(torch.int16))
        at += 6
    if extra:
        put(at, torch.randn(n, generator=gen, device=dev))
    return rec


def _hotspots(n, seed, extent, gen, dev):
    """20 Gaussian hot-spots at 100 times the background density over a slab
    50 m high (synth.hotspots on the device)."""
    rng = np.random.default_rng(seed)
    sig = rng.uniform(5.0, 40.0, 20)
    cx, cy = rng.uniform(0.1 * extent, 0.9 * extent, (2, 20))
    w = 100.0 * math.pi * sig ** 2
    edges = torch.tensor(np.concatenate([[extent * extent], w]).cumsum() / (extent * extent + w.sum()), device=dev)
    which = torch.searchsorted(edges, torch.rand(n, generator=gen, device=dev, dtype=torch.float64)).clamp(0, 20)
    spot = which > 0
    t = [torch.tensor(np.concatenate([[0.0], v]), device=dev)[which] for v in (sig, cx, cy)]
    u = [torch.rand(n, generator=gen, device=dev, dtype=torch.float64) for _ in range(3)]
    g = [torch.randn(n, generator=gen, device=dev, dtype=torch.float64) for _ in range(3)]
    x = torch.where(spot, t[1] + g[0] * t[0], u[0] * extent).clamp(0, extent)
    y = torch.where(spot, t[2] + g[1] * t[0], u[1] * extent).clamp(0, extent)
    z = torch.where(spot, (25.0 + g[2] * t[0] * 0.3).clamp(0, 50.0), u[2] * 50.0)
    return [(v / synth.SCALE).round().to(torch.int32) for v in (x, y, z)]


def _lattice(n, seed, extent, gen, dev):
    """Sites of a lattice whose pitch is the level-3 node spacing, each
    coordinate moved by 1-3 quantization units (synth.lattice)."""
    layers = max(1, -(-n // (1024 * 1024)))
    site = torch.randperm(1024 * 1024 * layers, generator=gen, device=dev)[:n]
    pitch = extent / 1024.0 / synth.SCALE
    out = []
    for idx in (site % 1024, (site // 1024) % 1024, site // (1024 * 1024)):
        step = torch.randint(1, 4, (n,), generator=gen, device=dev) * (torch.randint(0, 2, (n,), generator=gen, device=dev) * 2 - 1)
        out.append((idx.to(torch.float64) * pitch).round().to(torch.int32) + step.to(torch.int32))
    return out


_EXTRA_VLR = bytearray(54 + 192)
_EXTRA_VLR[2:11] = b"LASF_Spec"
struct.pack_into("<HH", _EXTRA_VLR, 18, 4, 192)
_EXTRA_VLR[54 + 2] = 9  # one float32
_EXTRA_VLR[54 + 4:54 + 9] = b"extra"


def _header(box, n, pdrf, rec_len, extra):
    lo, hi = box
    return synth.las_header(n, pdrf=pdrf, version_minor=4 if pdrf in (1, 3) else 2, record_length=rec_len, vlrs=bytes(_EXTRA_VLR) if extra else b"",
                            has_extra=extra, scale=(synth.SCALE,) * 3, offset=(0.0,) * 3,
                            bbox=sum(((hi[a] * synth.SCALE, lo[a] * synth.SCALE) for a in range(3)), ()), by_return=np.array([n, 0, 0, 0, 0]))


def _roomy(head):
    """The header of an image with its box half a quantum wider than the
    points: like the reference, the converter may refuse the outermost point
    of a box that is exact, by a rounding error."""
    head = bytearray(head)
    for at in (179, 195, 211):
        struct.pack_into("<d", head, at, struct.unpack_from("<d", head, at)[0] + 0.5 * struct.unpack_from("<d", head, 131)[0])
    return bytes(head)


def _pinned(img):
    img[:227] = torch.frombuffer(bytearray(_roomy(img[:227].numpy().tobytes())), dtype=torch.uint8)
    return img


def _cloud(case, seed):
    """(header bytes, records on the device) or a page-locked image."""
    n, cloud = case["points"], case["cloud"]
    if cloud == "terrain":
        return _pinned(synth_gpu.terrain(n, seed, case["extent"], case["pdrf"]))
    if cloud == "strips":
        return _pinned(synth_gpu.strips(n, seed, extent=case["extent"]))
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    extra = cloud == "hotspots"
    X, Y, Z = (_hotspots if extra else _lattice)(n, seed, case["extent"], gen, dev)
    rec = _write_columns(X, Y, Z, case["pdrf"], gen, extra)
    box = [[int(getattr(v, f)()) for v in (X, Y, Z)] for f in ("min", "max")]
    return _roomy(_header(box, n, case["pdrf"], rec.shape[1], extra)), rec


def _image(case, seed):
    """The file image in host memory, page-locked or not."""
    got = _cloud(case, seed)
    if isinstance(got, tuple):
        head, rec = got
        img = torch.empty(len(head) + rec.numel(), dtype=torch.uint8, pin_memory=True)
        img[:len(head)] = torch.frombuffer(bytearray(head), dtype=torch.uint8)
        img[len(head):].copy_(rec.view(-1))
        got = img
    return got.clone() if case.get("source") == "host" else got


# ------------------------------------------------------------ a LAZ writer
class _Symbols:
    """Adaptive model of n symbols."""

    def __init__(self, n):
        self.n, self.count, self.total, self.cycle = n, [1] * n, 0, n
        self.update()
        self.cycle = self.until = (n + 6) >> 1

    def update(self):
        self.total += self.cycle
        if self.total > 1 << 15:
            self.count = [(c + 1) >> 1 for c in self.count]
            self.total = sum(self.count)
        scale, s, dist = 0x80000000 // self.total, 0, []
        for c in self.count:
            dist.append((scale * s) >> 16)
            s += c
        self.dist = dist
        self.cycle = self.until = min((5 * self.cycle) >> 2, (self.n + 6) << 3)


class _Bit:
    """Adaptive model of one bit."""

    def __init__(self):
        self.zeros, self.count, self.prob, self.cycle, self.until = 1, 2, 1 << 12, 4, 4

    def update(self):
        self.count += self.cycle
        if self.count > 1 << 13:
            self.count, self.zeros = (self.count + 1) >> 1, (self.zeros + 1) >> 1
            if self.zeros == self.count:
                self.count += 1
        self.prob = (self.zeros * (0x80000000 // self.count)) >> 18
        self.cycle = self.until = min((5 * self.cycle) >> 2, 64)


class _Encoder:
    """The arithmetic coder: an interval [base, base + length)."""

    def __init__(self):
        self.out, self.base, self.length = bytearray(), 0, 0xFFFFFFFF

    def _settle(self):
        base, out = self.base, self.out
        if base >> 32:
            base &= 0xFFFFFFFF
            k = len(out) - 1
            while out[k] == 255:
                out[k] = 0
                k -= 1
            out[k] += 1
        while self.length < 1 << 24:
            out.append(base >> 24)
            base = (base << 8) & 0xFFFFFFFF
            self.length <<= 8
        self.base = base

    def symbol(self, m, s):
        if s == m.n - 1:
            x = m.dist[s] * (self.length >> 15)
            self.length -= x
        else:
            part = self.length >> 15
            x = m.dist[s] * part
            self.length = m.dist[s + 1] * part - x
        self.base += x
        if self.length < 1 << 24 or self.base >> 32:
            self._settle()
        m.count[s] += 1
        m.until -= 1
        if not m.until:
            m.update()

    def bit(self, m, s):
        x = m.prob * (self.length >> 13)
        if s:
            self.base += x
            self.length -= x
        else:
            self.length = x
            m.zeros += 1
        if self.length < 1 << 24 or self.base >> 32:
            self._settle()
        m.until -= 1
        if not m.until:
            m.update()

    def raw(self, v, bits):
        if bits > 19:
            self.raw(v & 0xFFFF, 16)
            v, bits = v >> 16, bits - 16
        self.length >>= bits
        self.base += v * self.length
        if self.length < 1 << 24 or self.base >> 32:
            self._settle()

    def finish(self):
        return bytes(self.out) + struct.pack(">I", self.base)


class _Residuals:
    """Integers coded as their distance from a prediction: its bit length by
    a model per context, then the value within that length."""

    def __init__(self, bits, contexts):
        self.bits, self.contexts = bits, [None] * contexts
        self.within = [None] * 33
        self.bit = _Bit()

    def code(self, enc, pred, real, ctx=0):
        """Returns the bit length, a context of the fields that follow."""
        half = 1 << (self.bits - 1)
        c = (real - pred + half) % (2 * half) - half
        k = (-c if c <= 0 else c - 1).bit_length()
        m = self.contexts[ctx]
        if m is None:
            m = self.contexts[ctx] = _Symbols(self.bits + 1)
        enc.symbol(m, k)
        if not k:
            enc.bit(self.bit, c)
            return 0
        if k == 32:
            return k
        v = c + (1 << k) - 1 if c < 0 else c - 1
        m = self.within[k]
        if m is None:
            m = self.within[k] = _Symbols(1 << min(k, 8))
        if k <= 8:
            enc.symbol(m, v)
        else:
            enc.symbol(m, v >> (k - 8))
            enc.raw(v & ((1 << (k - 8)) - 1), k - 8)
        return k


class _Median:
    """The middle of the last five values, as the format keeps it."""

    def __init__(self):
        self.v, self.high = [0] * 5, True

    def add(self, x):
        v = self.v
        if self.high:
            if x < v[2]:
                v[:] = sorted([v[0], v[1], x]) + [v[2], v[3]]
            else:
                if x < v[3]:
                    v[4], v[3] = v[3], x
                else:
                    v[4] = x
                self.high = False
        elif v[2] < x:
            v[:] = [v[1], v[2]] + sorted([v[3], v[4], x])
        else:
            if v[1] < x:
                v[0], v[1] = v[1], x
            else:
                v[0] = x
            self.high = True


# context of (number of returns, return number)
_RETURN_MAP = [[15, 14, 13, 12, 11, 10, 9, 8], [14, 0, 1, 3, 6, 10, 10, 9], [13, 1, 2, 4, 7, 11, 11, 10], [12, 3, 4, 5, 8, 12, 12, 11],
               [11, 6, 7, 8, 9, 13, 13, 12], [10, 10, 11, 12, 13, 14, 14, 13], [9, 10, 11, 12, 13, 14, 15, 14], [8, 9, 10, 11, 12, 13, 14, 15]]


def _scan(n, seed, pdrf):
    """n points of one flight segment: lines of 250 pulses 0.4 m apart, one
    to three returns per pulse, ground and vegetation. Columns of Python
    integers (coordinates in quanta, GPS time as the bits of a float64)."""
    rng = np.random.default_rng(seed)
    returns = rng.choice([1, 2, 3], n, p=[0.72, 0.2, 0.08])
    pulse = np.repeat(np.arange(n), returns)[:n]
    first = np.concatenate([[True], pulse[1:] != pulse[:-1]])
    nret = returns[pulse]
    ret = np.arange(n) - np.maximum.accumulate(np.where(first, np.arange(n), 0)) + 1
    line, step = pulse // 250, pulse % 250
    across = np.where(line % 2, 249 - step, step)
    x = across * 0.4 + rng.normal(0, 0.03, n)
    y = line * 0.5 + step * 0.002 + rng.normal(0, 0.03, n)
    ground = 60 + 4 * np.sin(x * 0.06) + 3 * np.cos(y * 0.045) + rng.normal(0, 0.03, n)
    z = ground + np.where(ret < nret, rng.uniform(1.0, 18.0, n), 0.0)
    intensity = np.clip(rng.normal(110, 22, n) / nret, 1, 255).astype(np.int64) * 16
    ticks = np.float64(3.0e5).view(np.int64) + (pulse + 20 * line) * 171_799
    ticks = ticks + np.where(first, rng.integers(-2, 3, n), 0)[np.maximum.accumulate(np.where(first, np.arange(n), 0))]
    shade = np.clip(rng.normal(120, 9, n)[pulse] + 20 * np.sin(x * 0.2), 0, 255).astype(np.int64)
    rgb = [np.clip(shade + d + rng.integers(-4, 5, n), 0, 255) * 256 for d in (6, 14, -20)]
    cols = dict(x=np.round(x * 1000), y=np.round(y * 1000), z=np.round(z * 1000), intensity=intensity, bits=ret | (nret << 3),
                cls=np.where(ret < nret, 5, np.where(rng.random(n) < 0.03, 6, 2)), angle=np.round((across - 125) * 0.12).astype(np.int64) & 255,
                gps=ticks, r=rgb[0], g=rgb[1], b=rgb[2])
    return {k: v.astype(np.int64).tolist() for k, v in cols.items()}


def _clamp8(v):
    return 0 if v < 0 else 255 if v > 255 else v


def _code_chunk(c, n, pdrf):
    """The points 1 .. n-1 of one chunk, coded (point 0 is stored raw)."""
    enc = _Encoder()
    changed, angle = _Symbols(64), [_Symbols(256), _Symbols(256)]
    by_bits, by_class = {}, {}
    ints, dx, dy, hz, gps = _Residuals(16, 4), _Residuals(32, 2), _Residuals(32, 22), _Residuals(32, 20), _Residuals(32, 9)
    mx, my = [_Median() for _ in range(16)], [_Median() for _ in range(16)]
    last_int, last_z = [0] * 16, [0] * 8
    zero_diff, multi = _Symbols(6), _Symbols(516)
    used, diff = _Symbols(128), [_Symbols(256) for _ in range(6)]
    x, y, z, intensity, bits, cls, ang, gpst = (c[k] for k in ("x", "y", "z", "intensity", "bits", "cls", "angle", "gps"))
    red, green, blue = c["r"], c["g"], c["b"]
    gps_step = 0
    symbol = enc.symbol
    for i in range(1, n):
        b, p = bits[i], i - 1
        r, nr = b & 7, (b >> 3) & 7
        m, lvl = _RETURN_MAP[nr][r], abs(nr - r)
        what = (b != bits[p]) << 5 | (intensity[i] != last_int[m]) << 4 | (cls[i] != cls[p]) << 3 | (ang[i] != ang[p]) << 2
        symbol(changed, what)
        if what & 32:
            t = by_bits.get(bits[p])
            if t is None:
                t = by_bits[bits[p]] = _Symbols(256)
            symbol(t, b)
        if what:
            if what & 16:
                ints.code(enc, last_int[m], intensity[i], m if m < 3 else 3)
                last_int[m] = intensity[i]
            if what & 8:
                t = by_class.get(cls[p])
                if t is None:
                    t = by_class[cls[p]] = _Symbols(256)
                symbol(t, cls[i])
            if what & 4:
                symbol(angle[(b >> 6) & 1], (ang[i] - ang[p]) & 255)
        one = nr == 1
        d = x[i] - x[p]
        kx = dx.code(enc, mx[m].v[2], d, one)
        mx[m].add(d)
        d = y[i] - y[p]
        ky = dy.code(enc, my[m].v[2], d, one + (kx & ~1 if kx < 20 else 20))
        my[m].add(d)
        kz = (kx + ky) // 2
        hz.code(enc, last_z[lvl], z[i], one + (kz & ~1 if kz < 18 else 18))
        last_z[lvl] = z[i]
        if pdrf in (1, 3):
            d = gpst[i] - gpst[p]
            if not gps_step:
                symbol(zero_diff, 1 if d else 0)
                if d:
                    gps.code(enc, 0, d, 0)
                    gps_step = d
            elif not d:
                symbol(multi, 511)
            else:
                k = int(round(d / gps_step))
                symbol(multi, k)
                gps.code(enc, k * gps_step, d, 1 if k == 1 else 2 if k < 10 else 3)
        if pdrf in (2, 3):
            # 8-bit colours in the high bytes: the low ones never change
            R, G, B = red[i] >> 8, green[i] >> 8, blue[i] >> 8
            r0, g0, b0 = red[p] >> 8, green[p] >> 8, blue[p] >> 8
            grey = R == G == B
            s = (R != r0) << 1 | (not grey) << 6
            if not grey:
                s |= (G != g0) << 3 | (B != b0) << 5
            symbol(used, s)
            if s & 2:
                symbol(diff[1], (R - r0) & 255)
            if s & 64:
                d = R - r0
                if s & 8:
                    symbol(diff[3], (G - _clamp8(d + g0)) & 255)
                if s & 32:
                    d += G - g0
                    symbol(diff[5], (B - _clamp8(int(d / 2) + b0)) & 255)
    return enc.finish()


def _laz(case, seed):
    """A LAZ image: every chunk is the same coded flight segment laid at
    another place and time (a chunk's first point is stored raw, the others
    as differences), the last one cut short."""
    n, chunk, pdrf = case["points"], min(case["chunk"], case["points"]), case["pdrf"]
    c = _scan(chunk, seed, pdrf)
    coded = _code_chunk(c, chunk, pdrf)
    count = -(-n // chunk)
    rng = np.random.default_rng(seed + 1)
    lines = max(c["y"]) + 1000
    side = max(1, int(math.ceil(math.sqrt(count * lines / 100_000))))
    body = bytearray()
    lo, hi = [2 ** 31] * 3, [-2 ** 31] * 3
    for k in range(count):
        sx = (k % side) * 100_000 + int(rng.integers(0, 400))
        sy = (k // side) * lines + int(rng.integers(0, 400))
        first = struct.pack("<3iHBBBBH", c["x"][0] + sx, c["y"][0] + sy, c["z"][0], c["intensity"][0], c["bits"][0], c["cls"][0], c["angle"][0], 0, 17)
        if pdrf in (1, 3):
            first += struct.pack("<q", c["gps"][0] + k * 10 ** 9)
        if pdrf in (2, 3):
            first += struct.pack("<3H", c["r"][0], c["g"][0], c["b"][0])
        body += first + coded
        for a, (col, s) in enumerate((("x", sx), ("y", sy), ("z", 0))):
            lo[a], hi[a] = min(lo[a], min(c[col]) + s), max(hi[a], max(c[col]) + s)
    size = len(body) // count
    table, sizes, last = _Encoder(), _Residuals(32, 2), 0
    for _ in range(count):
        sizes.code(table, last, size, 1)
        last = size
    items = [(6, 20)] + [(7, 8)] * (pdrf in (1, 3)) + [(8, 6)] * (pdrf in (2, 3))
    vlr = struct.pack("<HHBBHIIqqH", 2, 0, 3, 4, 3, 0, chunk, -1, -1, len(items)) + b"".join(struct.pack("<HHH", t, s, 2) for t, s in items)
    record = bytearray(54)
    record[2:16] = b"laszip encoded"
    struct.pack_into("<HH", record, 18, 22204, len(vlr))
    head = bytearray(synth.las_header(n, pdrf=pdrf, version_minor=2, record_length=REC_LEN[pdrf], vlrs=bytes(record) + vlr, has_extra=True,
                                      scale=(synth.SCALE,) * 3, offset=(0.0,) * 3,
                                      bbox=sum(((hi[a] * synth.SCALE, lo[a] * synth.SCALE) for a in range(3)), ()),
                                      by_return=np.array([n, 0, 0, 0, 0])))
    head[104] |= 0x80
    at = len(head) + 8 + len(body)
    return _roomy(head) + struct.pack("<q", at) + bytes(body) + struct.pack("<II", 0, count) + table.finish() + bytes(8)


# ------------------------------------------------------------------ passes
_contexts = {}


def _context(group=0):
    """The contexts a long-running program keeps: one for each part size."""
    if group not in _contexts:
        _contexts[group] = pc.Context(group_points=group)
    return _contexts[group]


class _Bytes:
    """A buffer of a pcg_result, kept alive with it."""

    def __init__(self, owner, ptr, size, device=False):
        self.owner = owner
        face = {"data": (ptr, False), "shape": (size,), "typestr": "|u1", "version": 3}
        if device:
            self.__cuda_array_interface__ = face
        else:
            self.__array_interface__ = face


class _Owned:
    """A pcg_result, freed when the last view of its buffers goes."""

    def __init__(self):
        self.res = pc._Result()

    def __del__(self):
        pc.load_library().pcg_result_free(ctypes.byref(self.res))

    def octree(self, on_device):
        """octree.bin in pieces, as tensors over the library's buffers."""
        r = self.res
        if on_device:
            ptr = ctypes.cast(r.octree, ctypes.c_void_p).value
            return [torch.as_tensor(_Bytes(self, ptr, r.octree_size, True), device="cuda")]
        parts = [r.octree_parts[k] for k in range(r.num_octree_parts)]
        return [torch.from_numpy(np.asarray(_Bytes(self, ctypes.cast(p.data, ctypes.c_void_p).value, p.size))) for p in parts if p.size]


class _Files:
    """Where a program keeps a conversion's three files: buffers with room
    for the largest it expects, zero past their end. octree.bin stays in the
    library's buffer when it comes in one piece of a size known beforehand
    (every point once); else its pieces are put back to back."""

    def __init__(self, points, bpp, method, pieces=False, device="cpu"):
        self.size = points * bpp
        self.whole = not pieces and method != "poisson_average"
        self.octree = None if self.whole else torch.zeros(self.size * 4 if method == "poisson_average" else self.size, dtype=torch.uint8,
                                                          device=device).fill_(0)
        self.hierarchy = np.zeros(22 * (points // 100 + 8192), np.uint8)
        self.metadata = np.zeros(16384, np.uint8)

    def take(self, owned, on_device=False):
        r = owned.res
        for buf, ptr, size in ((self.hierarchy, r.hierarchy, r.hierarchy_size), (self.metadata, r.metadata, r.metadata_size)):
            if size > buf.size:
                raise ValueError("a result larger than expected")
            ctypes.memmove(buf.ctypes.data, ptr, size)
        pieces = owned.octree(on_device)
        if self.whole and len(pieces) == 1:
            octree = pieces[0]
        else:
            octree, at = self.octree, 0
            for p in pieces:
                octree[at:at + p.numel()].copy_(p)
                at += p.numel()
        return {"octree": octree, "hierarchy": self.hierarchy, "metadata": self.metadata}


class _Call:
    """A pcg_job and what it points to."""

    def __init__(self, method, images, header=None, records=None, attributes=""):
        self.keep = [images, records]
        if records is not None:
            self.job = pc.Context._job(header, method, "cloud", "", self.keep, device_records=records.data_ptr(), flags=pc.OCTREE_ON_DEVICE)
        else:
            las = [i if isinstance(i, bytes) else (i.data_ptr(), i.numel()) for i in images]
            self.job = pc.Context._job(las if len(las) > 1 else las[0], method, "cloud", "", self.keep,
                                       attributes=attributes.split(",") if attributes else None)


def _sizes(case):
    """Points and sampler of every job of a queue: sizes spread over their
    logarithm, samplers mixed 60 / 30 / 10 %."""
    lo, hi, jobs = case["smallest"], case["largest"], case["jobs"]
    for k in range(jobs):
        n = int(lo * (hi / lo) ** (((k * 7) % jobs) / max(jobs - 1, 1))) | 1
        yield n, ("poisson", "poisson", "poisson_average", "poisson", "poisson_average", "poisson", "poisson", "random", "poisson_average", "poisson")[k % 10]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "queue":
        jobs = [_Call(m, [_pinned(synth_gpu.terrain(n, seed * 31 + k, case["extent"], 2 + k % 2))]) for k, (n, m) in enumerate(_sizes(case))]
        files = [_Files(n, REC_LEN[2 + k % 2] + 1, m) for k, (n, m) in enumerate(_sizes(case))]
        return {"queue": jobs, "files": files, "ctx": _context()}
    if kind == "tiles":
        call = _Call(case["method"], [_roomy(t[:227]) + t[227:] for t in synth.tiles(case["points"], seed, case["extent"])], attributes=case["attributes"])
    elif kind == "laz":
        call = _Call(case["method"], [_laz(case, seed)])
    elif case["source"] == "resident":
        got = _cloud(case, seed)
        if not isinstance(got, tuple):  # a page-locked image: its records go to the device
            at = 375 if int(got[25]) >= 4 else 227
            got = bytes(got[:at].numpy()), got[at:].cuda()
        call = _Call(case["method"], [], *got)
    else:
        call = _Call(case["method"], [_image(case, seed)])
    on_device = case.get("source") == "resident"
    files = _Files(case["points"], _record_bytes(case)[1], case["method"], pieces=kind == "parts", device="cuda" if on_device else "cpu")
    return {"call": call, "files": files, "ctx": _context(case.get("group", 0)), "on_device": on_device}


def run(state):
    lib, ctx = pc.load_library(), state["ctx"]
    if "queue" in state:
        ids = []
        for call in state["queue"]:
            ids.append(ctypes.c_uint64())
            _check(ctx, lib.pcg_submit(ctx._h, ctypes.byref(call.job), ctypes.byref(ids[-1])))
        out = []
        for i, files in zip(ids, state["files"]):
            owned = _Owned()
            _check(ctx, lib.pcg_wait(ctx._h, i, ctypes.byref(owned.res)))
            out.append(files.take(owned))
        return out
    owned = _Owned()
    _check(ctx, lib.pcg_convert(ctx._h, ctypes.byref(state["call"].job), ctypes.byref(owned.res)))
    return state["files"].take(owned, state["on_device"])


def _check(ctx, status):
    if status:
        raise ctx._err(status)


def _record_bytes(case):
    """Bytes of an input record and of an output point."""
    if case["kind"] == "tiles":
        # filtered: position, rgb, classification, intensity; else every
        # attribute of the four formats and their extra bytes
        return sum(REC_LEN[f] for f in synth.TILE_FORMATS) / 4 + 3, 21 if case["attributes"] else 43
    if case["kind"] == "laz":
        return 12, REC_LEN[case["pdrf"]] + 1  # about 12 coded bytes a point
    rec = HOTSPOT_REC if case["cloud"] == "hotspots" else REC_LEN[case["pdrf"]]
    return rec, rec + 1  # the two return numbers take a byte each


def work(case):
    """Records read once, octree.bin written once. The sampler that averages
    writes a point into its node and into the nodes above that accept it:
    measured 3.1 times the points on the hot-spots, 1.7 on the others."""
    keep = 1.0
    if case.get("method") == "poisson_average":
        keep = 3.1 if case.get("cloud") == "hotspots" else 1.7
    if case["kind"] == "queue":
        jobs = [(n, m, REC_LEN[2 + k % 2]) for k, (n, m) in enumerate(_sizes(case))]
    else:
        jobs = [(case["points"], case["method"], None)]
    total = 0.0
    for n, method, rec in jobs:
        rec, out = (rec, rec + 1) if rec else _record_bytes(case)
        total += n * (rec + out * (1.7 if method == "poisson_average" and keep == 1.0 else keep))
    return {"bytes": total, "flops": 0}

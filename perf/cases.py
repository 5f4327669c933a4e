"""Performance cases of the clipping library, each through its public Python entry points.

A case says what a program clips: one pair of rings, one base against many overlays, or a batch of
independent pairs, as rings or as areas with their gradients.  ``prepare`` makes the inputs, ``run``
is one call (or one forward and backward) as a user's program makes it, ``work`` counts the input
and output bytes, and ``exact`` gives the same rings, areas and gradients from a plain FP64
computation on edge crossings (no segment tree, no linked lists), for general position.

Shapes: a "star" has angle k in its own sector of the circle and radius R (0.5 + 0.5 u); a
"jagged" ring has the same angles and eight octaves of periodic value noise on its radius.
The library's classifier compares signed areas with an absolute 1e-9, so rings of many vertices
are large (pixels or metres), where no area of theirs is near that.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

PKG = Path(__file__).resolve().parent.parent / "segment-tree-based-clipping_gb300"
if str(PKG) not in sys.path:
    sys.path.insert(0, str(PKG))

import sbclip  # noqa: E402

TWO_PI = 2.0 * math.pi
STAR_MOST = 12_000  # vertices of a plain star; larger rings are jagged
BASE_CELLS = 6000  # lowest noise octave of a base with many overlays


def _radius(n):
    return 1.0 if n <= 64 else 1e3 if n <= 4_096 else 1e5


# ------------------------------------------------------------------ cases
def listed():
    return [
        # the smallest call: two dozen vertices against eighteen, host arrays, where latency is all
        {"name": "pair_24_18", "kind": "pair", "nb": 24, "nc": 18, "host": True},
        # the reference's `seg base overlay` at its everyday size (ten thousand vertices)
        {"name": "pair_10k_8k", "kind": "pair", "nb": 10_000, "nc": 8_000, "host": True},
        # a large map layer against a small one, odd sizes, arrays already on the device
        {"name": "pair_300k_15k_device", "kind": "pair", "nb": 300_007, "nc": 15_013, "host": False},
        # the headline: one million vertices against one million, host arrays in and out
        {"name": "pair_1m_1m", "kind": "pair", "nb": 1_000_000, "nc": 1_000_000, "host": True},
        # the reference's multi-overlay command line: one tree over a base and its overlays
        {"name": "tree_30k_x5", "kind": "tree", "nb": 30_011, "overlays": 5, "lo": 2_003, "hi": 9_001},
        # union mode on a batch of uneven mid-size pairs, rings back on the host
        {"name": "union_rings_400", "kind": "batch_rings", "pairs": 400, "lo": 8, "hi": 700, "union": True},
        # one base layer against thousands of small overlays, rings back on the host
        {"name": "overlays_rings_4000", "kind": "pairwise_rings", "nb": 200_000, "overlays": 4_000, "lo": 4, "hi": 5_000},
        # the same job in a training step: areas and gradients, device arrays
        {"name": "overlays_grad_10000", "kind": "pairwise_grad", "nb": 200_000, "overlays": 10_000, "lo": 4, "hi": 5_000},
        # a training step on many small pairs (boxes, cells, glyphs): one recorded graph per step
        {"name": "small_graph_65536", "kind": "batch_graph", "pairs": 65_536, "lo": 4, "hi": 64},
        # a minibatch of the same, forward and backward as separate calls on device arrays
        {"name": "small_grad_512", "kind": "batch_grad", "pairs": 512, "lo": 4, "hi": 64, "large": 0, "host": False},
        # very uneven pairs with one large one among them, host arrays in and out
        {"name": "uneven_grad_12000", "kind": "batch_grad", "pairs": 12_000, "lo": 3, "hi": 2_048, "large": 50_000, "host": True},
        # polygons with holes and islands, forward and backward
        {"name": "holed_grad_1500", "kind": "holed_grad", "pairs": 1_500, "lo": 16, "hi": 160, "holes": 2, "islands": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges, sizes spread over their logarithm."""
    kind = rng.choice(["pair", "pair", "tree", "batch_rings", "pairwise_rings", "pairwise_grad",
                       "batch_graph", "batch_grad", "batch_grad", "holed_grad"])
    if kind == "pair":
        return {"kind": kind, "nb": _log_int(rng, 12, 900_000), "nc": _log_int(rng, 12, 900_000),
                "host": rng.random() < 0.5}
    if kind == "tree":
        lo = _log_int(rng, 50, 4_000)
        return {"kind": kind, "nb": _log_int(rng, 500, 100_000), "overlays": rng.randint(2, 9),
                "lo": lo, "hi": lo * rng.randint(2, 5) + 1}
    if kind == "batch_rings":
        return {"kind": kind, "pairs": _log_int(rng, 20, 600), "lo": rng.randint(3, 20),
                "hi": _log_int(rng, 40, 700), "union": rng.random() < 0.5}
    if kind == "pairwise_rings":
        return {"kind": kind, "nb": _log_int(rng, 2_500, 200_000), "overlays": _log_int(rng, 30, 4_000),
                "lo": rng.randint(3, 40), "hi": _log_int(rng, 100, 5_000)}
    if kind == "pairwise_grad":
        return {"kind": kind, "nb": _log_int(rng, 2_500, 200_000), "overlays": _log_int(rng, 30, 9_000),
                "lo": rng.randint(3, 40), "hi": _log_int(rng, 100, 5_000)}
    if kind == "batch_graph":
        return {"kind": kind, "pairs": _log_int(rng, 64, 60_000), "lo": rng.randint(3, 12),
                "hi": rng.randint(16, 64)}
    if kind == "batch_grad":
        return {"kind": kind, "pairs": _log_int(rng, 16, 9_000), "lo": rng.randint(3, 24),
                "hi": _log_int(rng, 32, 2_048), "large": rng.choice([0, 0, 20_000]),
                "host": rng.random() < 0.5}
    islands = rng.randint(0, 2)
    return {"kind": kind, "pairs": _log_int(rng, 16, 1_500), "lo": 16, "hi": rng.randint(24, 160),
            "holes": rng.randint(max(1, islands), 3), "islands": islands}


# ------------------------------------------------------------------ inputs
def _offsets(sizes):
    return np.concatenate([[0], np.cumsum(np.asarray(sizes, np.int64))])


def _stars(rng, sizes, centres, radii):
    """Packed plain stars (n >= 3 vertices each, counter-clockwise)."""
    off = _offsets(sizes)
    seg = np.repeat(np.arange(len(sizes)), sizes)
    k = np.arange(off[-1]) - off[seg]
    th = TWO_PI * (k + rng.uniform(0.1, 0.9, off[-1])) / np.asarray(sizes)[seg]
    r = np.asarray(radii)[seg] * (0.5 + 0.5 * rng.random(off[-1]))
    xy = np.stack([r * np.cos(th), r * np.sin(th)], axis=1)
    return xy + np.asarray(centres, np.float64)[seg], off


def _jagged(rng, n, R, centre=(0.0, 0.0), cells=None):
    th = TWO_PI * (np.arange(n) + rng.uniform(0.1, 0.9, n)) / n
    g = np.zeros(n)
    low = cells or max(8, n // 166)
    for o in range(8):
        cells = low << o
        lattice = rng.uniform(-1.0, 1.0, cells + 1)
        lattice[-1] = lattice[0]
        t = th * (cells / TWO_PI)
        k = np.minimum(t.astype(np.int64), cells - 1)
        f = t - k
        s = f * f * (3.0 - 2.0 * f)
        g += (lattice[k] * (1.0 - s) + lattice[k + 1] * s) * 0.5 ** o
    r = np.maximum(R * (1.0 + 0.3 * g), 0.2 * R)
    return np.stack([centre[0] + r * np.cos(th), centre[1] + r * np.sin(th)], axis=1)


def _ring(rng, n, R, overlay):
    """A base ring about the origin, or an overlay ring a quarter of a radius off it."""
    centre = (0.25 * R, 0.1 * R) if overlay else (0.0, 0.0)
    return _jagged(rng, n, R, centre) if n > STAR_MOST else _stars(rng, [n], [centre], [R])[0]


def _sizes(rng, lo, hi, n):
    return np.clip(np.exp(rng.uniform(math.log(lo), math.log(hi + 1), n)).astype(np.int64), lo, hi)


def _overlays(rng, base, lo, hi, n):
    """Plain stars over a large base: log-uniform sizes and radii, centres in the base's box."""
    centres = rng.uniform(base.min(axis=0), base.max(axis=0), (n, 2))
    radii = _radius(len(base)) * np.exp(rng.uniform(math.log(0.003), math.log(0.06), n))
    return _stars(rng, _sizes(rng, lo, hi, n), centres, radii)


def _pairs(rng, lo, hi, n, large=0):
    """Packed pairs of stars, overlay centres within half a radius; with `large`, one pair of
    jagged rings of that size in the middle."""
    R = _radius(hi)
    out = []
    for overlay in (False, True):
        sizes = _sizes(rng, lo, hi, n)
        centres = rng.uniform(-0.5 * R, 0.5 * R, (n, 2)) if overlay else np.zeros((n, 2))
        xy, off = _stars(rng, sizes, centres, np.full(n, R))
        if large:
            at = n // 2
            ring = _ring(rng, large, _radius(large), overlay)
            xy = np.concatenate([xy[:off[at]], ring, xy[off[at]:]])
            off = np.concatenate([off[:at + 1], off[at:] + large])
        out += [xy, off]
    return out


def _holed(rng, case):
    """Packed polygons with holes (clockwise) and islands in the first holes: outer radius
    0.7..1, holes on a circle of radius 0.4.  Also the component offsets."""
    n, holes, islands = case["pairs"], case["holes"], case["islands"]
    out = []
    for overlay in (False, True):
        outer = _sizes(rng, case["lo"], case["hi"], n)
        inner = np.maximum(outer // 4, 16)
        kinds = ["outer"] + [k for h in range(holes) for k in (["hole", "island"] if h < islands else ["hole"])]
        sizes = np.stack([outer if k == "outer" else inner for k in kinds], axis=1).reshape(-1)
        comp = _offsets(sizes)
        seg = np.repeat(np.arange(len(sizes)), sizes)
        k = np.arange(comp[-1]) - comp[seg]
        cw = np.tile([kind == "hole" for kind in kinds], n)
        k = np.where(cw[seg], sizes[seg] - 1 - k, k)
        th = TWO_PI * (k + rng.uniform(0.05, 0.95, comp[-1])) / sizes[seg]
        span = {"outer": (0.7, 1.0), "hole": (0.12, 0.2), "island": (0.04, 0.08)}
        lo = np.tile([span[q][0] for q in kinds], n)
        hi = np.tile([span[q][1] for q in kinds], n)
        r = lo[seg] + (hi - lo)[seg] * rng.random(comp[-1])
        at = np.cumsum([q == "hole" for q in kinds]) - 1  # the hole of each component
        a = rng.uniform(0.0, TWO_PI, n)[:, None] + TWO_PI * at[None, :] / holes
        d = np.where(np.asarray(kinds) == "outer", 0.0, 0.4)
        c = np.stack([d * np.cos(a), d * np.sin(a)], axis=-1)
        c = (c + (rng.uniform(-0.5, 0.5, (n, 1, 2)) if overlay else 0.0)).reshape(-1, 2)
        xy = np.stack([r * np.cos(th), r * np.sin(th)], axis=1) + c[seg]
        out += [_radius(case["hi"]) * xy, comp[:: len(kinds)].copy(), comp]
    return out


def _placed(case, seed, xys, group):
    """The polygons turned, scaled and moved, each group (a pair, or a base with its overlays) by
    a placement of its own that the seed draws: all coordinates differ between seeds, and the
    result's rings have the same sizes."""
    rng = np.random.default_rng(seed)
    n = 1 + max(int(g.max()) for g in group)
    angle, scale = rng.uniform(0.0, TWO_PI, n), rng.uniform(0.8, 1.25, n)
    a, b = scale * np.cos(angle), scale * np.sin(angle)
    move = rng.uniform(-0.5, 0.5, (n, 2))
    return [np.stack([a[g] * xy[:, 0] - b[g] * xy[:, 1], b[g] * xy[:, 0] + a[g] * xy[:, 1]], axis=1) + move[g]
            for xy, g in zip(xys, group)]


def _inputs(case, seed):
    """The polygons of a case as NumPy arrays: shapes that the case fixes, placed by the seed."""
    data = _shapes(case)
    kind = case["kind"]
    if kind in ("pair", "tree", "pairwise_rings", "pairwise_grad"):
        at = [0, 1] if kind != "tree" else [0]
        xys = [data[i] for i in at] + (data[1] if kind == "tree" else [])
        xys = _placed(case, seed, xys, [np.zeros(len(v), np.int64) for v in xys])
        return [xys[0], xys[1:]] if kind == "tree" else xys + data[2:]
    per = 3 if kind == "holed_grad" else 2
    off = (data[1], data[per + 1])
    data[0], data[per] = _placed(case, seed, (data[0], data[per]),
                                 [np.repeat(np.arange(len(o) - 1), np.diff(o)) for o in off])
    if kind == "batch_rings":
        return [[v[o[i]:o[i + 1]] for i in range(len(o) - 1)] for v, o in ((data[0], data[1]), (data[2], data[3]))]
    return data


def _shapes(case):
    numbers = [v for v in case.values() if isinstance(v, int)]
    rng = np.random.default_rng(numbers)
    kind = case["kind"]
    if kind == "pair":
        R = _radius(max(case["nb"], case["nc"]))
        return [_ring(rng, case["nb"], R, False), _ring(rng, case["nc"], R, True)]
    if kind == "tree":
        R = _radius(max(case["nb"], case["hi"]))
        sizes = _sizes(rng, case["lo"], case["hi"], case["overlays"])
        return [_jagged(rng, case["nb"], R),
                [_jagged(rng, int(n), R * rng.uniform(0.3, 1.0), rng.uniform(-0.5 * R, 0.5 * R, 2)) for n in sizes]]
    if kind in ("pairwise_rings", "pairwise_grad"):
        base = _jagged(rng, case["nb"], _radius(case["nb"]), cells=BASE_CELLS)
        return [base, *_overlays(rng, base, case["lo"], case["hi"], case["overlays"])]
    if kind == "batch_rings":
        return _pairs(rng, case["lo"], case["hi"], case["pairs"])
    if kind == "holed_grad":
        return _holed(rng, case)
    return _pairs(rng, case["lo"], case["hi"], case["pairs"], case.get("large", 0))


def _upstream(rng_seed, n):
    """The gradient that reaches the areas from a loss."""
    return np.random.default_rng([rng_seed, 1]).uniform(-1.0, 1.0, n)


# ------------------------------------------------------------------ states and passes
_clippers = {}


def _clipper(union=False):
    """A program keeps one library context for all its calls."""
    if union not in _clippers:
        _clippers[union] = sbclip.Clipper(0, union=union)
    return _clippers[union]


class _GraphState(dict):
    """A recorded step with the context that it belongs to."""

    def __del__(self):
        self["graph"].close()
        self["clipper"].close()


class _DeviceArray:
    """Library-owned device memory as the CUDA array interface describes it."""

    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _on_device(ptr, shape, typestr, dtype):
    if ptr is None or 0 in shape:
        return torch.zeros(shape, dtype=dtype, device="cuda")
    return torch.as_tensor(_DeviceArray(ptr, shape, typestr), device="cuda")


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def prepare(case, seed):
    kind = case["kind"]
    data = _inputs(case, seed)
    if kind in ("tree", "batch_rings", "pairwise_rings") or (kind in ("pair", "batch_grad") and case["host"]):
        state = {"kind": kind + ("_host" if kind in ("pair", "batch_grad") else ""), "in": data,
                 "clipper": _clipper(bool(case.get("union")))}
        if kind == "batch_grad":
            state["up"] = _upstream(seed, len(data[1]) - 1)
        return state
    dev = [_cuda(a) for a in data]
    state = {"kind": kind, "in": dev, "clipper": _clipper()}
    if kind == "pair":
        torch.cuda.synchronize()
        return state
    n = case["overlays"] if kind == "pairwise_grad" else len(data[1]) - 1
    bxy, cxy = (dev[0], dev[3]) if kind == "holed_grad" else (dev[0], dev[1 if kind == "pairwise_grad" else 2])
    state["up"] = _cuda(_upstream(seed, n))
    state["area"] = torch.zeros(n, dtype=torch.float64, device="cuda")
    state["status"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    state["grad_b"], state["grad_c"] = torch.zeros_like(bxy), torch.zeros_like(cxy)
    torch.cuda.synchronize()
    if kind == "batch_graph":
        state["clipper"] = sbclip.Clipper(0)
        ptr = [a.data_ptr() for a in dev]
        state["graph"] = state["clipper"].area_graph(
            n, *ptr, state["up"].data_ptr(), state["grad_b"].data_ptr(), state["grad_c"].data_ptr(),
            state["area"].data_ptr(), state["status"].data_ptr())
        return _GraphState(state)
    return state


def _flat(rings):
    """A ring list as one vertex array and the ring sizes."""
    return (np.concatenate(rings) if rings else np.zeros((0, 2)),
            np.array([len(r) for r in rings], np.int64))


def run(state):
    kind, c, data = state["kind"], state["clipper"], state["in"]
    if kind == "pair_host":
        return c.clip_pair_flat(data[0], data[1], copy=False)
    if kind == "pair":
        nr, nv, off, xy = c.clip_pair_device(data[0].data_ptr(), len(data[0]), data[1].data_ptr(), len(data[1]))
        return (_on_device(off, (nr + 1 if nr else 0,), "<i4", torch.int32),
                _on_device(xy, (nv, 2), "<f8", torch.float64))
    if kind == "tree":
        return [_flat(rings) for rings in c.clip(data[0], data[1])]
    if kind == "batch_rings":
        rings, status = c.clip_batch(data[0], data[1])
        return (*_flat([r for pair in rings for r in pair]), np.array([len(p) for p in rings]), status)
    if kind == "pairwise_rings":
        return c.clip_pairwise_flat(data[0], data[1], data[2], copy=False)
    if kind == "batch_grad_host":
        area, status = c.area_forward_packed(*data)
        grad_b, grad_c = c.area_backward_packed(*data, state["up"])
        return area, status, grad_b, grad_c
    area, status, gb, gc = state["area"], state["status"], state["grad_b"], state["grad_c"]
    if kind == "batch_graph":
        state["graph"].launch()
    elif kind == "batch_grad":
        ptr = [a.data_ptr() for a in data]
        n = len(data[1]) - 1
        c.area_forward_device(n, *ptr, area.data_ptr(), status.data_ptr())
        c.area_backward_device(n, *ptr, state["up"].data_ptr(), gb.data_ptr(), gc.data_ptr())
    elif kind == "pairwise_grad":
        job = (data[0].data_ptr(), len(data[0]), len(data[2]) - 1, data[1].data_ptr(), data[2].data_ptr())
        c.pairwise_area_device(*job, area.data_ptr(), status.data_ptr())
        c.pairwise_area_backward_device(*job, state["up"].data_ptr(), gb.data_ptr(), gc.data_ptr())
    else:
        bxy, boff, bcomp, cxy, coff, ccomp = data
        job = (len(boff) - 1, bxy.data_ptr(), boff.data_ptr(), cxy.data_ptr(), coff.data_ptr(),
               bcomp.data_ptr(), len(bcomp) - 1, ccomp.data_ptr(), len(ccomp) - 1)
        c.area_forward_components_device(*job, area.data_ptr(), status.data_ptr())
        c.area_backward_components_device(*job, state["up"].data_ptr(), gb.data_ptr(), gc.data_ptr())
    return area, status, gb, gc


def _mean_size(case):
    lo, hi = case["lo"], case["hi"]
    return lo if hi <= lo else (hi - lo) / math.log(hi / lo)


def work(case):
    """Input coordinates read once, results written once: a ring result holds about as many
    vertices as its smaller polygon, gradients as many as the inputs."""
    kind = case["kind"]
    if kind == "pair":
        return {"bytes": 16 * (case["nb"] + case["nc"] + min(case["nb"], case["nc"])), "flops": 0}
    if kind == "tree":
        return {"bytes": 16 * (case["nb"] + 2 * case["overlays"] * _mean_size(case)), "flops": 0}
    if kind.startswith("pairwise"):
        total = case["overlays"] * _mean_size(case)
        twice = 2 if kind == "pairwise_grad" else 1
        return {"bytes": 16 * (twice * case["nb"] + 2 * total) + 20 * case["overlays"], "flops": 0}
    total = 2 * case["pairs"] * _mean_size(case) + 2 * case.get("large", 0)
    if kind == "holed_grad":
        total *= 1 + (case["holes"] + case["islands"]) / 4
    if kind == "batch_rings":
        return {"bytes": 16 * 1.5 * total + 20 * case["pairs"], "flops": 0}
    return {"bytes": 32 * total + 36 * case["pairs"], "flops": 0}


# ------------------------------------------------------------------ exact values
class _Side:
    """One side's components: vertices, each component's first vertex, each component's pair."""

    def __init__(self, xy, comp, pair, device):
        self.xy = torch.as_tensor(np.ascontiguousarray(xy), device=device)
        self.first = torch.as_tensor(comp[:-1], device=device)
        self.size = torch.as_tensor(np.diff(comp), device=device)
        self.pair = None if pair is None else torch.as_tensor(pair, device=device)  # None: all pairs
        self.of = torch.repeat_interleave(torch.arange(len(comp) - 1, device=device), self.size)
        v = torch.arange(len(self.xy), device=device)
        self.succ = torch.where(v + 1 == (self.first + self.size)[self.of], self.first[self.of], v + 1)

    def edge(self, e):
        return self.xy[e], self.xy[self.succ[e]]

    def blocks(self, width):
        """Blocks of up to `width` consecutive edges of one component: first edge, count, box."""
        per = (self.size + width - 1) // width
        at = torch.repeat_interleave(torch.arange(len(per), device=per.device), per)
        k = torch.arange(len(at), device=per.device) - (torch.cumsum(per, 0) - per)[at]
        start = self.first[at] + k * width
        count = torch.minimum(self.size[at] - k * width, torch.full_like(k, width))
        e = torch.minimum(start[:, None] + torch.arange(width, device=per.device), (start + count - 1)[:, None])
        p = torch.stack([self.xy[e], self.xy[self.succ[e]]], 0)
        return start, count, at, p.amin((0, 2)), p.amax((0, 2))


def _cross(a, b):
    return a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]


def _block_pairs(B, C, b, c):
    """Pairs of blocks of the same pair whose boxes overlap."""
    bi, ci = [], []
    if B.pair is None:
        step = max(1, 30_000_000 // max(1, len(b[0])))
        for s in range(0, len(c[0]), step):
            lo, hi = c[3][s:s + step, None], c[4][s:s + step, None]
            hit = ((b[3] <= hi) & (b[4] >= lo)).all(-1).nonzero()
            ci.append(hit[:, 0] + s)
            bi.append(hit[:, 1])
    else:  # blocks are in pair order on both sides
        pb, pc = B.pair[b[2]], C.pair[c[2]].contiguous()
        lo, hi = torch.searchsorted(pc, pb), torch.searchsorted(pc, pb, right=True)
        step = max(1, 20_000_000 // max(1, int((hi - lo).max())))
        for s in range(0, len(pb), step):
            n = (hi - lo)[s:s + step]
            i = torch.repeat_interleave(torch.arange(s, s + len(n), device=n.device), n)
            j = torch.arange(len(i), device=n.device) - (torch.cumsum(n, 0) - n)[i - s] + lo[i]
            ok = ((b[3][i] <= c[4][j]) & (b[4][i] >= c[3][j])).all(-1)
            bi.append(i[ok])
            ci.append(j[ok])
    return torch.cat(bi), torch.cat(ci)


def _crossings(B, C, width):
    """(pair, base edge, s, overlay edge, t, base enters) of every proper crossing."""
    b, c = B.blocks(width), C.blocks(width)
    bi, ci = _block_pairs(B, C, b, c)
    lane = torch.arange(width, device=bi.device)
    found = []
    step = max(1, (1 << 25) // (width * width))
    for s in range(0, max(1, len(bi)), step):
        i, j = bi[s:s + step], ci[s:s + step]
        eb, ec = b[0][i][:, None] + lane, c[0][j][:, None] + lane
        ub, uc = lane < b[1][i][:, None], lane < c[1][j][:, None]
        eb, ec = torch.where(ub, eb, b[0][i][:, None]), torch.where(uc, ec, c[0][j][:, None])
        (b1, b2), (c1, c2) = B.edge(eb), C.edge(ec)
        lo, hi = torch.minimum(b1, b2), torch.maximum(b1, b2)
        ok = ub[:, :, None] & uc[:, None, :]
        for x in (0, 1):
            ok &= (lo[:, :, None, x] <= torch.maximum(c1, c2)[:, None, :, x]) & (hi[:, :, None, x] >= torch.minimum(c1, c2)[:, None, :, x])
        k, p, q = ok.nonzero(as_tuple=True)
        eb, ec = eb[k, p], ec[k, q]
        (b1, b2), (c1, c2) = B.edge(eb), C.edge(ec)
        s1, s2 = _cross(c2 - c1, b1 - c1), _cross(c2 - c1, b2 - c1)
        t1, t2 = _cross(b2 - b1, c1 - b1), _cross(b2 - b1, c2 - b1)
        ok = ((s1 > 0) != (s2 > 0)) & ((t1 > 0) != (t2 > 0))
        found.append((C.pair[C.of[ec]][ok], eb[ok], (s1 / (s1 - s2))[ok], ec[ok], (t1 / (t1 - t2))[ok], (s2 > 0)[ok]))
    return [torch.cat(v) for v in zip(*found)]


def _lex(*keys):
    order = torch.arange(len(keys[0]), device=keys[0].device)
    for k in reversed(keys):
        order = order[torch.argsort(k[order], stable=True)]
    return order


def _next(group):
    """Cyclic successor within runs of equal `group` (sorted)."""
    n = len(group)
    i = torch.arange(n, device=group.device)
    first = torch.searchsorted(group, group)
    return torch.where((i + 1 < n) & (torch.roll(group, -1) == group), i + 1, first)


def _inside(points, pair, S):
    """Whether each point lies in the polygon of its pair on side S (even-odd)."""
    out = torch.zeros(len(points), dtype=torch.bool, device=points.device)
    ep = torch.arange(len(S.xy), device=points.device) if S.pair is None else S.pair[S.of]
    n_edges = len(S.xy)
    if S.pair is None:
        lo, hi = torch.zeros_like(pair), torch.full_like(pair, n_edges)
    else:
        lo, hi = torch.searchsorted(ep, pair), torch.searchsorted(ep, pair, right=True)
    step = max(1, 20_000_000 // max(1, int((hi - lo).max()) if len(pair) else 1))
    for s in range(0, len(points), step):
        n = (hi - lo)[s:s + step]
        i = torch.repeat_interleave(torch.arange(s, s + len(n), device=n.device), n)
        e = torch.arange(len(i), device=n.device) - (torch.cumsum(n, 0) - n)[i - s] + lo[i]
        (a, b), p = S.edge(e), points[i]
        odd = ((a[:, 1] > p[:, 1]) != (b[:, 1] > p[:, 1])) & (
            (_cross(b - a, p - a) > 0) == (b[:, 1] > a[:, 1]))
        out[s:s + step] = torch.zeros(len(n), dtype=torch.int64, device=n.device).index_add_(0, i - s, odd.long()) % 2 == 1
    return out


def _intersect(B, C, npairs, width):
    """The boundary of every pair's intersection as edge pieces.

    A piece is (side, edge, from, to, pair, sign): pieces of the base inside the overlay and of the
    overlay inside the base.  The library starts a ring at its first crossing along the base and
    walks the base from there inside the overlay, so a ring that starts where the base leaves the
    overlay is walked backwards: its sign is -1.  Also the rings: (first crossing, crossing ids,
    ring of each crossing, next crossing, flipped)."""
    dev = B.xy.device
    pair, eb, s, ec, t, enters = _crossings(B, C, width)
    o = _lex(pair, eb, s)
    pair, eb, s, ec, t, enters = (v[o] for v in (pair, eb, s, ec, t, enters))
    n = len(pair)
    ids = torch.arange(n, device=dev)
    next_b = _next(pair * len(B.first) + B.of[eb]) if n else ids
    oc = _lex(C.of[ec], ec, t)
    next_c = ids.clone()
    if n:
        next_c[oc] = oc[_next(C.of[ec][oc])]
    nxt = torch.where(enters, next_b, next_c)
    ring, jump = ids.clone(), nxt.clone()
    for _ in range(max(1, n).bit_length()):
        ring = torch.minimum(ring, ring[jump])
        jump = jump[jump]
    sign = torch.where(enters[ring], 1.0, -1.0).to(torch.float64) if n else torch.zeros(0, dtype=torch.float64, device=dev)
    pieces = []
    for S, e, u, mine in ((B, eb, s, enters), (C, ec, t, ~enters)):
        i = ids[mine]
        j = nxt[i]
        cnt = torch.remainder(e[j] - e[i], S.size[S.of[e[i]]])
        cnt = torch.where((cnt == 0) & (u[j] < u[i]), S.size[S.of[e[i]]], cnt)
        # cnt whole or partial edges follow the one that the piece starts on
        rep = torch.repeat_interleave(torch.arange(len(i), device=dev), cnt + 1)
        k = torch.arange(len(rep), device=dev) - (torch.cumsum(cnt + 1, 0) - cnt - 1)[rep]
        c0 = S.first[S.of[e[i]]][rep]
        edge = c0 + torch.remainder(e[i][rep] - c0 + k, S.size[S.of[e[i]]][rep])
        lo = torch.where(k == 0, u[i][rep], torch.zeros_like(u[i][rep]))
        hi = torch.where(k == cnt[rep], u[j][rep], torch.ones_like(lo))
        # components that cross nothing count whole where they lie inside
        if S.pair is None:
            lone = torch.ones(npairs, dtype=torch.bool, device=dev)
            lone[pair] = False
            lp = lone.nonzero()[:, 0]
            comp = torch.zeros_like(lp)
        else:
            lone = torch.ones(len(S.first), dtype=torch.bool, device=dev)
            lone[S.of[e]] = False
            comp = lone.nonzero()[:, 0]
            lp = S.pair[comp]
        ins = _inside(S.xy[S.first[comp]], lp, C if S is B else B)
        comp, lp = comp[ins], lp[ins]
        rep2 = torch.repeat_interleave(torch.arange(len(comp), device=dev), S.size[comp])
        k2 = torch.arange(len(rep2), device=dev) - (torch.cumsum(S.size[comp], 0) - S.size[comp])[rep2]
        edge = torch.cat([edge, S.first[comp][rep2] + k2])
        zero = torch.zeros(len(rep2), dtype=torch.float64, device=dev)
        pieces.append((S, edge, torch.cat([lo, zero]), torch.cat([hi, zero + 1]),
                       torch.cat([pair[i][rep], lp[rep2]]), torch.cat([sign[i][rep], zero + 1]),
                       torch.cat([i[rep], torch.full_like(rep2, -1)]), torch.cat([k, k2])))
    return pieces, (ring, nxt, enters)


def _areas(B, C, npairs, up, width):
    """Areas and their gradients.  Moving a piece of edge (v1, v2) sweeps the integral of its
    normal velocity, which is linear along the edge."""
    pieces, _ = _intersect(B, C, npairs, width)
    area = torch.zeros(npairs, dtype=torch.float64, device=B.xy.device)
    grads = []
    for S, edge, lo, hi, pair, sign, _, _ in pieces:
        v1, v2 = S.edge(edge)
        d = v2 - v1
        area.index_add_(0, pair, 0.5 * sign * (hi - lo) * _cross(v1, d))
        normal = torch.stack([d[:, 1], -d[:, 0]], 1) * (sign * up[pair])[:, None]
        w2 = 0.5 * (hi * hi - lo * lo)
        g = torch.zeros_like(S.xy)
        g.index_add_(0, edge, normal * (hi - lo - w2)[:, None])
        g.index_add_(0, S.succ[edge], normal * w2[:, None])
        grads.append(g)
    return area, grads[0], grads[1]


def _rings(B, C, npairs, width):
    """Ring vertices in the library's order, packed: rings by first crossing, each from the
    vertex after that crossing, vertices in line with both neighbours left out."""
    pieces, (ring, nxt, enters) = _intersect(B, C, npairs, width)
    dev = B.xy.device
    n = len(ring)
    # vertices of each crossing's piece: the crossing itself, then the starts of the further edges
    at = torch.cat([p[6] for p in pieces])
    k = torch.cat([p[7] for p in pieces])
    pair = torch.cat([p[4] for p in pieces])
    xy = torch.cat([p[0].edge(p[1])[0] + p[2][:, None] * (p[0].edge(p[1])[1] - p[0].edge(p[1])[0]) for p in pieces])
    cnt = torch.zeros(n, dtype=torch.int64, device=dev)
    cnt.index_add_(0, at[at >= 0], torch.ones_like(at[at >= 0]))
    # vertices from each crossing to its ring's end, and on the whole ring
    left = _suffix(cnt, nxt, ring)
    total = left[ring]
    pos, key = k.clone(), torch.full_like(at, n)
    on = at >= 0
    of = at[on]
    pos[on] += (total - left)[of]
    flip = (~enters)[ring[of]] & (pos[on] > 0)
    pos[on] = torch.where(flip, total[of] - pos[on], pos[on])
    pos[on] = torch.where(pos[on] == 0, total[of], pos[on])  # the first crossing closes the ring
    key[on] = ring[of]
    o = _lex(pair, key, pos)
    xy, key, pair = xy[o], key[o], pair[o]
    g = pair * (n + 1) + key
    i = torch.arange(len(g), device=dev)
    first = torch.searchsorted(g, g)
    last = torch.searchsorted(g, g, right=True) - 1
    before = xy[torch.where(i == first, last, i - 1)]
    after = xy[torch.where(i == last, first, i + 1)]
    return xy[_cross(xy - before, after - before).abs() >= 1e-9], pair


def _suffix(cnt, nxt, ring):
    """Sum of cnt from each element to the end of its cycle cut before the cycle's `ring` element."""
    n = len(cnt)
    ids = torch.arange(n, device=cnt.device)
    end = nxt == ring
    jump = torch.where(end, ids, nxt)
    total = torch.where(end, torch.zeros_like(cnt), cnt)
    for _ in range(max(1, n).bit_length()):
        total = total + total[jump]
        jump = jump[jump]
    return total + cnt[jump]


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if case.get("union"):
        return None  # the pieces above are the intersection's
    data = _inputs(case, seed)
    if kind in ("pair", "tree"):
        found = []
        for c in ([data[1]] if kind == "pair" else data[1]):
            sides = [_Side(v, np.array([0, len(v)]), np.zeros(1, np.int64), device) for v in (data[0], c)]
            sides[0].pair = None
            found.append(_rings(*sides, 1, 64)[0])
        return [None, found[0]] if kind == "pair" else [(xy, None) for xy in found]
    if kind == "batch_rings":
        packed = [np.concatenate(v) for v in data]
        offs = [_offsets([len(p) for p in v]) for v in data]
        n = len(data[0])
        return [_rings(*(_Side(v, o, np.arange(n), device) for v, o in zip(packed, offs)), n, 32)[0], None, None, None]
    if kind.startswith("pairwise"):
        n = case["overlays"]
        B = _Side(data[0], np.array([0, len(data[0])]), None, device)
        C = _Side(data[1], data[2], np.arange(n), device)
        if kind == "pairwise_rings":
            return [None, None, _rings(B, C, n, 64)[0], None]
        area, gb, gc = _areas(B, C, n, torch.as_tensor(_upstream(seed, n), device=device), 64)
        return [area, None, gb, gc]
    if kind == "holed_grad":
        bxy, boff, bcomp, cxy, coff, ccomp = data
        n = len(boff) - 1
        per = (len(bcomp) - 1) // n
        B, C = (_Side(v, comp, np.repeat(np.arange(n), per), device) for v, comp in ((bxy, bcomp), (cxy, ccomp)))
    else:
        bxy, boff, cxy, coff = data
        n = len(boff) - 1
        B, C = _Side(bxy, boff, np.arange(n), device), _Side(cxy, coff, np.arange(n), device)
    area, gb, gc = _areas(B, C, n, torch.as_tensor(_upstream(seed, n), device=device), 32)
    return [area, None, gb, gc]

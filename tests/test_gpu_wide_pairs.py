"""Pairs whose rows A9-A18 run on a block instead of a warp: rings equal to the
oracle's, bit for bit, for plain crossings (the block's own labelling and
tracing) and for touching and overlapping edges (its first warp's serial
steps), in both modes and on either side of the size rule."""
import numpy as np
import pytest

import oracle_py
import sbclip
import sbclip_gen as gen
from conftest import rings_equal

pytestmark = pytest.mark.gpu


def comb(teeth, y0, y1, x0, up, flat):
    """A comb along x: a bar and `teeth` slanted teeth with flat tips at y1
    (or at flat[i] of the way).  No vertical edge."""
    s = 1.0 if up else -1.0
    v = []
    for i in range(teeth):
        tip = y0 + (y1 - y0) * flat[i % len(flat)]
        v += [(x0 + i, y0), (x0 + i + 0.13, tip), (x0 + i + 0.57, tip), (x0 + i + 0.71, y0)]
    bar = [(x0 + teeth + 0.31, y0 - s * 1.0), (x0 - 0.83, y0 - s * 1.0)]
    p = np.array(v + bar)
    return p if not up else p[::-1].copy()


def want(base, ov, union):
    return oracle_py.rings_of(oracle_py.clip(base, [ov], union=union)["overlays"][0])


@pytest.fixture(scope="module", params=[False, True], ids=["intersection", "union"])
def mode(request):
    c = sbclip.Clipper(0, union=request.param)
    yield c, request.param
    c.close()


def test_plain_crossings(mode):
    """Records on both sides of the block's line (512) and up to 20,000, an
    overlay that starts inside the base and one that starts outside, one of
    either orientation, a whole base inside an overlay."""
    cl, union = mode
    base = gen.star(2500, 71, R=100.0)
    ovs = [gen.star(n, 900 + n, centre=(x, 7.0), R=r)
           for n, x, r in ((3, 0.0, 90.0), (64, 20.0, 40.0), (127, 30.0, 60.0), (300, 10.0, 80.0),
                           (301, -35.0, 95.0), (1200, 25.0, 100.0), (2400, 3.0, 100.0),
                           (700, 0.0, 30.0), (40, 0.0, 1000.0), (50, 900.0, 20.0))]
    ovs.append(ovs[5][::-1].copy())
    # with and without the rule that hands a few large pairs to the pipeline
    few, few_status = cl.clip_pairwise(base, ovs)
    cl.set_pairwise_split(1 << 30)
    try:
        rings, status = cl.clip_pairwise(base, ovs)
        assert cl.pairwise_info()["big_pairs"] == 0
    finally:
        cl.set_pairwise_split(32768)
    assert (status == 0).all() and (few_status == 0).all()
    for got, same, o in zip(rings, few, ovs):
        assert rings_equal(got, want(base, o, union)) and rings_equal(got, same)


def test_overlaps_and_touches(mode):
    """Flat tips of the two combs meet along edges (delayed crossings and
    bounces): the block leaves these pairs' serial steps to one warp."""
    cl, union = mode
    base = comb(420, 0.0, 1.0, 0.0, True, [1.0, 0.7, 1.0, 1.0])
    ovs = [comb(n, 2.0, 1.0, x, False, f)
           for n, x, f in ((400, 0.2937, [1.0, 1.4]), (300, 40.4143, [1.0, 1.3, 1.0]),
                           (410, 3.6189, [1.5, 1.2, 1.45]), (8, 5.2711, [1.0]))]
    rings, status = cl.clip_pairwise(base, ovs)
    for got, o, st in zip(rings, ovs, status):
        try:
            ref = want(base, o, union)
        except oracle_py.OracleError:
            assert st != 0
            continue
        assert st == 0 and rings_equal(got, ref)


@pytest.mark.parametrize("shared", [False, True], ids=["apart", "shared_x"])
def test_pairwise_general_position_and_not(mode, shared):
    """Overlays in general position, and not: vertices and edges on the base,
    a vertex of the base, an x value twice, a crossing within the classifier's
    epsilon of a vertex, several records on one edge, the whole base in the
    result (more ring vertices than a pair's first arena), none.  With a base
    whose x values are apart and one that has two alike.  Rings as the
    oracle's; areas to 1e-12 of the rings' absolute terms and gradients to
    1e-11 of their largest entry (FP64 sums in another order)."""
    import area_grad
    torch = pytest.importorskip("torch")
    cl, union = mode
    base = gen.star(1500, 171, R=100.0)
    if shared:
        base[700, 0] = base[3, 0]
    v, e = base[100], (base[200] + base[201]) / 2
    out = np.array([170.0, 60.0])
    ovs = [gen.star(n, 700 + n, centre=(x, 3.0), R=r)
           for n, x, r in ((3, 1.0, 80.0), (33, 9.0, 60.0), (90, 20.0, 90.0), (400, -9.0, 100.0),
                           (40, 0.0, 1000.0), (30, 0.0, 5.0), (20, 900.0, 20.0))]
    ovs += [np.array([v, out, out + [3.0, 60.0]]), np.array([e, out, out + [3.0, 60.0]]),
            np.array([base[300], base[301], out]), np.array([v + 1e-10, out, out + [3.0, 60.0]]),
            np.array([[-150.0, -1.3], [150.0, 2.1], [150.0, 9.7], [-140.0, 5.2]]),
            np.array([[-150.0, -1.3], [150.0, 2.1], [145.0, 9.7], [-140.0, 5.2]]),
            ovs[2][::-1].copy()]
    rings, status = cl.clip_pairwise(base, ovs)
    seen = []
    for i, (got, o, st) in enumerate(zip(rings, ovs, status)):
        try:
            ref = oracle_py.clip(base, [o], union=union)["overlays"][0]
        except oracle_py.OracleError:
            assert st != 0
            continue
        assert st == 0 and rings_equal(got, oracle_py.rings_of(ref)), i
        seen.append((i, ref))
    assert len(seen) >= 10
    ga = np.zeros(len(ovs))
    ga[[i for i, _ in seen]] = np.random.default_rng(3).uniform(0.5, 2.0, len(seen))
    cxy, coff = sbclip.pack_polygons(ovs)
    tb, tc, to, tg = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (base, cxy, coff, ga))
    ta, ts = torch.zeros_like(tg), torch.zeros(len(ovs), dtype=torch.int32, device="cuda")
    job = (tb.data_ptr(), len(base), len(ovs), tc.data_ptr(), to.data_ptr())
    cl.pairwise_area_device(*job, ta.data_ptr(), ts.data_ptr())
    tgb, tgc = torch.zeros_like(tb), torch.zeros_like(tc)
    cl.pairwise_area_backward_device(*job, tg.data_ptr(), tgb.data_ptr(), tgc.data_ptr())
    area, gb, gc = ta.cpu().numpy(), tgb.cpu().numpy(), np.split(tgc.cpu().numpy(), coff[1:-1])
    sum_b = np.zeros_like(base)
    for i, ref in seen:
        rs = oracle_py.rings_of(ref)
        scale = sum(float(np.abs(r).max() ** 2) * len(r) for r in rs) + 1e-300
        assert abs(area[i] - area_grad.shoelace(rs)) <= 1e-12 * scale, i
        _, rb, rc = area_grad.gradient_of_rings(base, ovs[i], rs, ref["uniq_b"], ref["uniq_c"],
                                                ref["uniq_t"], ref["isect_xy"])
        top = ga[i] * max(np.abs(rb).max(), np.abs(rc).max(), 1e-300)
        assert np.abs(gc[i] - ga[i] * rc).max() <= 1e-11 * top, i
        sum_b += ga[i] * rb
    assert np.abs(gb - sum_b).max() <= 1e-11 * max(np.abs(sum_b).max(), 1e-300)


# ------------------------------------------------------------------ batches
def batch_pairs():
    """Either side of the wide rule (16,384 edge pairs) and of the front's
    shared-memory sort (1,024 edges), edge groups of 32 with a remainder, more
    crossings than the first pass has room for, coordinates on a grid (shared
    x values, vertical edges), overlapping edges, either orientation, one
    polygon inside the other, disjoint ones."""
    rng = np.random.default_rng(11)
    out = []
    for i, (nb, nc) in enumerate(((128, 128), (128, 129), (4, 4096), (4096, 5), (160, 161), (511, 513),
                                  (512, 513), (1023, 33), (1000, 1100), (2048, 64), (2048, 2047))):
        off = rng.uniform(-40.0, 40.0, 2)
        out.append((gen.star(nb, 500 + i, R=100.0), gen.star(nc, 600 + i, centre=off, R=100.0)))
    out.append((out[5][0], out[5][1][::-1].copy()))
    out.append((gen.star(300, 41, R=100.0), gen.star(200, 42, R=10.0)))
    out.append((gen.star(300, 43, R=10.0), gen.star(200, 44, centre=(1.0, 0.0), R=900.0)))
    out.append((gen.star(300, 45, R=10.0), gen.star(200, 46, centre=(500.0, 0.0), R=9.0)))
    for i in range(3):
        b, c = gen.star(240, 51 + i, R=60.0), gen.star(180, 61 + i, centre=(9.0, -4.0), R=60.0)
        out.append((np.round(b * 4) / 4, np.round(c * 4) / 4))
    out.append((comb(90, 0.0, 1.0, 0.0, True, [1.0, 0.7, 1.0]), comb(80, 2.0, 1.0, 0.2937, False, [1.0, 1.4])))
    out.append((comb(90, 0.0, 1.0, 0.0, True, [1.0, 0.7, 1.0]), comb(80, 2.0, 1.0, 3.1441, False, [1.5, 1.3])))
    out.append((gen.star(3, 71), gen.star(4, 72)))
    return out


def test_batch_rings(mode):
    cl, union = mode
    pairs = batch_pairs()
    rings, status = cl.clip_batch([b for b, _ in pairs], [c for _, c in pairs])
    seen = 0
    for (b, c), got, st in zip(pairs, rings, status):
        try:
            ref = want(b, c, union)
        except oracle_py.OracleError:
            assert st != 0
            continue
        assert st == 0 and rings_equal(got, ref), (len(b), len(c))
        seen += 1
    assert seen >= len(pairs) - 4


def test_batch_area_and_gradient(clipper):
    """Areas to 1e-12 of the sum of the rings' absolute terms and gradients to
    1e-11 of their largest entry (both sides sum FP64 terms, here in another
    order), the same bits twice."""
    import area_grad
    pairs = []
    for b, c in batch_pairs():
        try:
            pairs.append((b, c, oracle_py.clip(b, [c])["overlays"][0]))
        except oracle_py.OracleError:
            pass
    bases, ovs = [p[0] for p in pairs], [p[1] for p in pairs]
    ga = np.random.default_rng(7).uniform(0.5, 2.0, len(pairs))
    area, status = clipper.area_forward(bases, ovs)
    gb, gc = clipper.area_backward(bases, ovs, ga)
    gb2, gc2 = clipper.area_backward(bases, ovs, ga)
    assert (status == 0).all()
    for p, (b, c, o) in enumerate(pairs):
        rings = oracle_py.rings_of(o)
        ref = area_grad.shoelace(rings)
        scale = sum(float(np.abs(r).max() ** 2) * len(r) for r in rings) + 1e-300
        assert abs(area[p] - ref) <= 1e-12 * scale
        _, rb, rc = area_grad.gradient_of_rings(b, c, rings, o["uniq_b"], o["uniq_c"], o["uniq_t"], o["isect_xy"])
        top = ga[p] * max(np.abs(rb).max(), np.abs(rc).max(), 1e-300)
        assert np.abs(gb[p] - ga[p] * rb).max() <= 1e-11 * top, (len(b), len(c))
        assert np.abs(gc[p] - ga[p] * rc).max() <= 1e-11 * top, (len(b), len(c))
        assert np.array_equal(gb[p], gb2[p]) and np.array_equal(gc[p], gc2[p])


def test_batch_rule_on_either_side(clipper):
    """More than 1,024 pairs above 4,096 edge pairs stay on warps, fewer run on
    blocks: the same rings, and areas to the rounding of a sum in another
    order."""
    pairs = gen.small_pairs(1030, seed=4700, lo=70, hi=75)
    bases, ovs = [b for b, _ in pairs], [c for _, c in pairs]
    many, st = clipper.clip_batch(bases, ovs)
    a_many, _ = clipper.area_forward(bases, ovs)
    assert (st == 0).all()
    few = [clipper.clip_batch(bases[i:i + 103], ovs[i:i + 103])[0] for i in range(0, 1030, 103)]
    few = [r for part in few for r in part]
    a_few = np.concatenate([clipper.area_forward(bases[i:i + 103], ovs[i:i + 103])[0] for i in range(0, 1030, 103)])
    assert all(rings_equal(x, y) for x, y in zip(many, few))
    assert np.abs(a_many - a_few).max() <= 1e-13
    for i in (0, 511, 1029):
        assert rings_equal(many[i], want(bases[i], ovs[i], False))


def test_general_position_and_not(mode):
    """Batches that mix pairs in general position with pairs that are not, by
    one reason each: a vertex on an edge, a shared vertex, overlapping edges,
    an x value of two vertices, a ring vertex in line with its neighbours, a
    crossing within the classifier's epsilon of a vertex.  Every pair as the
    oracle has it, in one batch and alone."""
    cl, union = mode
    sq = np.array([[0.0, 0.1], [4.0, 0.0], [4.1, 4.0], [0.2, 4.2]])
    cases = [
        (sq, sq + [1.7, 2.3]),
        (sq, np.array([[2.0, 0.05], [6.0, 1.1], [5.0, 3.3]])),            # vertex on an edge
        (sq, np.array([[4.0, 0.0], [7.0, 1.3], [5.0, 3.7]])),             # shared vertex
        (sq, np.array([[1.0, 0.075], [3.0, 0.025], [3.3, 2.0], [1.2, 2.1]])),  # overlapping edge
        (np.array([[0.0, 0.0], [4.0, 0.0], [4.0, 4.0], [0.0, 4.0]]), sq + [1.7, 2.3]),  # shared x
        (np.array([[0.0, 0.1], [1.0, 0.1 + 1e-10], [2.0, 0.1], [4.1, 4.0], [0.3, 4.2]]), sq + [-1.3, 1.9]),
        (sq, np.array([[2.0, 0.05 + 1e-10], [6.0, 1.1], [5.0, 3.3]])),
        (gen.star(60, 5), gen.star(50, 6, centre=(0.2, 0.1))),
        (gen.star(60, 5), gen.star(50, 6, centre=(0.2, 0.1))[::-1].copy()),
    ]
    rings, status = cl.clip_batch([b for b, _ in cases], [c for _, c in cases])
    for (b, c), got, st in zip(cases, rings, status):
        alone, st1 = cl.clip_batch([b], [c])
        assert st1[0] == st and rings_equal(alone[0], got)
        try:
            ref = want(b, c, union)
        except oracle_py.OracleError:
            assert st != 0
            continue
        assert st == 0 and rings_equal(got, ref)


@pytest.mark.parametrize("n,holes,islands", [(16, 1, 0), (40, 2, 1), (150, 3, 2), (700, 5, 5)])
def test_components_in_general_position(mode, n, holes, islands):
    """Polygons with holes and islands on a warp (small) and on a block (wide):
    rings as the oracle's."""
    cl, union = mode
    bases = [gen.holed(n, 30 + i, holes=holes, islands=islands) for i in range(6)]
    ovs = [gen.holed(n - (n > 16), 60 + i, centre=(0.11 * i, 0.07), holes=holes, islands=islands) for i in range(6)]
    rings, status = cl.clip_batch_components(bases, ovs)
    assert (status == 0).all()
    for b, c, got in zip(bases, ovs, rings):
        o = oracle_py.clip_components(b, c, union=union)["overlays"][0]
        assert rings_equal(got, oracle_py.rings_of(o))


def with_points(poly, edges, where):
    """poly with a point on each listed edge, `where` of the way (in line up to
    rounding)."""
    out = []
    for i, v in enumerate(poly):
        out.append(v)
        if i in edges:
            w = poly[(i + 1) % len(poly)]
            out += [v + t * (w - v) for t in where]
    return np.array(out)


@pytest.mark.parametrize("n", [12, 45, 300, 700])
def test_ring_vertices_in_line(mode, n):
    """Vertices in line with their neighbours, which the reference removes: one
    on an edge, on many, two and three in a row, the ring's first vertex, on
    edges with crossings, whole rings; on warps and on blocks, one component and several,
    one base against many overlays.  Rings as the oracle's."""
    cl, union = mode
    b = gen.star(n, 210 + n, R=50.0)
    cases = []
    for k, (edges, where) in enumerate((((1,), (0.4,)), (range(0, n, 3), (0.37,)), ((2, 7), (0.3, 0.8)),
                                        ((0, n - 1), (0.55,)), (range(n), (0.5,)),
                                        ((4, 5), (0.2, 0.5, 0.9)))):
        c = gen.star(n - k, 300 + n + k, centre=(4.1 + k, -2.3), R=45.0)
        cases.append((with_points(b, edges, where), c))
        cases.append((np.roll(with_points(b, edges, where), 2, axis=0), with_points(c, edges, where)))
    for k, deep in enumerate((1e-6, 4e-6, 3e-5)):  # a corner just across an edge: a sliver of a ring
        v, w = b[3 + k], b[4 + k]
        t = (w - v) / np.hypot(*(w - v))
        inward = np.array([-t[1], t[0]])
        tip = (v + w) / 2 + deep * inward
        cases.append((b, np.array([tip, tip - inward * 30.0 + 0.1 * t, tip - inward * 29.0 - 0.2 * t])))
        cases.append((b, np.array([tip - inward * 29.0 - 0.2 * t, tip + deep * t, tip - deep * t,
                                   tip - inward * 30.0 + 0.1 * t])))

    def expected(x, c, st):
        try:
            return want(x, c, union)
        except oracle_py.OracleError:
            assert st != 0
            return None

    rings, status = cl.clip_batch([x for x, _ in cases], [x for _, x in cases])
    for (x, c), got, st in zip(cases, rings, status):
        ref = expected(x, c, st)
        assert ref is None or (st == 0 and rings_equal(got, ref))
    for x in (cases[0][0], cases[3][1], cases[4][0]):
        ovs = [c for _, c in cases]
        rings, status = cl.clip_pairwise(x, ovs)
        for c, got, st in zip(ovs, rings, status):
            ref = expected(x, c, st)
            assert ref is None or (st == 0 and rings_equal(got, ref))
        comps = [[x, x * 0.5 + [300.3, 0.7]]] * 3
        others = [[ovs[0]], [ovs[3], ovs[0] + [299.1, 1.3]], [ovs[5]]]
        rings, status = cl.clip_batch_components(comps, others)
        for c, got, st in zip(others, rings, status):
            try:
                o = oracle_py.clip_components(comps[0], c, union=union)["overlays"][0]
            except oracle_py.OracleError:
                assert st != 0
                continue
            assert st == 0 and rings_equal(got, oracle_py.rings_of(o))


def test_device_arrays_aligned_to_a_double(clipper):
    """Coordinates that start 8 bytes past a 16-byte boundary: the same areas
    and gradients, from every engine that takes device arrays (the pairwise
    gradients to 1e-13 of the largest: atomic sums of a few terms)."""
    torch = pytest.importorskip("torch")

    def on_device(x, shift):
        x = torch.from_numpy(np.ascontiguousarray(x, dtype=np.float64)).cuda()
        t = torch.zeros(x.numel() + 1, dtype=torch.float64, device="cuda")[shift:][:x.numel()]
        t.copy_(x.reshape(-1))
        assert t.data_ptr() % 16 == 8 * shift
        return t

    base = gen.star(700, 81, R=100.0)
    ovs = [gen.star(n, 800 + n, centre=(x, 3.0), R=80.0) for n, x in ((5, 1.0), (60, 9.0), (600, -20.0))]
    cxy, coff = sbclip.pack_polygons(ovs)
    bxy, boff = sbclip.pack_polygons([base] * len(ovs))
    tco, tbo = torch.from_numpy(coff).cuda(), torch.from_numpy(boff).cuda()
    got = []
    for shift in (0, 1):
        tb, tc, tbb = on_device(base, shift), on_device(cxy, shift), on_device(bxy, shift)
        tg = torch.ones(len(ovs), dtype=torch.float64, device="cuda")
        ta, ta2 = torch.zeros_like(tg), torch.zeros_like(tg)
        ts = torch.zeros(len(ovs), dtype=torch.int32, device="cuda")
        gb, gc, gb2, gc2 = (on_device(np.zeros(x.numel()), shift) for x in (tb, tc, tbb, tc))
        job = (tb.data_ptr(), len(base), len(ovs), tc.data_ptr(), tco.data_ptr())
        clipper.pairwise_area_device(*job, ta.data_ptr(), ts.data_ptr())
        clipper.pairwise_area_backward_device(*job, tg.data_ptr(), gb.data_ptr(), gc.data_ptr())
        job = (len(ovs), tbb.data_ptr(), tbo.data_ptr(), tc.data_ptr(), tco.data_ptr())
        clipper.area_forward_device(*job, ta2.data_ptr(), ts.data_ptr())
        clipper.area_backward_device(*job, tg.data_ptr(), gb2.data_ptr(), gc2.data_ptr())
        counts = clipper.clip_pair_device(tb.data_ptr(), len(base), tc.data_ptr(), len(ovs[0]))
        got.append([x.cpu().numpy() for x in (ta, ta2, gb, gc, gb2, gc2)] + [np.array(counts[:2])])
    for i, (x, y) in enumerate(zip(*got)):
        if i in (2, 3):
            assert np.abs(x - y).max() <= 1e-13 * np.abs(x).max()
        else:
            assert np.array_equal(x, y), i


@pytest.mark.parametrize("sy", [1e-25, 1e-3, 1e12, 1e37, 1e39, 1e42])
def test_heights_near_and_beyond_float(mode, sy):
    """Heights at the ends of float's range and past it, where the float tests
    must keep every candidate: rings as the oracle's."""
    cl, union = mode
    scale = np.array([1.0, sy])
    pairs = [(gen.star(n, 20 + n, R=100.0) * scale, gen.star(m, 30 + m, centre=(7.0, 3.0), R=90.0) * scale)
             for n, m in ((9, 7), (40, 33), (200, 150), (700, 300))]
    pairs += [(b, c * np.array([1.0, -1e-6])) for b, c in pairs]
    for clip in (lambda: cl.clip_batch([b for b, _ in pairs], [c for _, c in pairs]),
                 lambda: [sum(x, []) for x in zip(*[tuple(map(list, cl.clip_pairwise(b, [c]))) for b, c in pairs])]):
        rings, status = clip()
        for (b, c), got, st in zip(pairs, rings, status):
            try:
                ref = want(b, c, union)
            except oracle_py.OracleError:
                assert st != 0
                continue
            assert st == 0 and rings_equal(got, ref)


def test_mixed_batch_on_two_streams_and_recorded(clipper):
    """A batch of small and wide pairs, whose kernels run side by side: the
    recorded step gives the bits of the separate calls, and again on new
    coordinates, on the context's stream and on a caller's."""
    torch = pytest.importorskip("torch")
    pairs = [p for p in batch_pairs() if len(p[0]) + len(p[1]) < 2500] + gen.small_pairs(60, seed=77, lo=4, hi=40)
    (bxy, boff), (cxy, coff) = (sbclip.pack_polygons([p[k] for p in pairs]) for k in (0, 1))
    n = len(pairs)
    tb, tbo, tc, tco = (torch.from_numpy(x).cuda() for x in (bxy, boff, cxy, coff))
    ga = torch.linspace(0.5, 2.0, n, dtype=torch.float64, device="cuda")
    args = (n, tb.data_ptr(), tbo.data_ptr(), tc.data_ptr(), tco.data_ptr())

    def separate(stream=None):
        area, st = torch.zeros_like(ga), torch.zeros(n, dtype=torch.int32, device="cuda")
        gb, gc = torch.zeros_like(tb), torch.zeros_like(tc)
        torch.cuda.synchronize()
        clipper.area_forward_device(*args, area.data_ptr(), st.data_ptr(), stream)
        clipper.area_backward_device(*args, ga.data_ptr(), gb.data_ptr(), gc.data_ptr(), stream)
        torch.cuda.synchronize()
        return [x.cpu().numpy() for x in (area, st, gb, gc)]

    def same(x, y):
        return all(np.array_equal(a, b) for a, b in zip(x, y))

    first = separate()
    own = torch.cuda.Stream()
    assert same(first, separate(own.cuda_stream))
    out = [torch.zeros_like(x) for x in (ga, ga.to(torch.int32), tb, tc)]
    g = clipper.area_graph(*args, ga.data_ptr(), out[2].data_ptr(), out[3].data_ptr(), out[0].data_ptr(),
                           out[1].data_ptr())
    torch.cuda.synchronize()
    for scale in (1.0, 1.25):
        tb.copy_(torch.from_numpy(bxy * scale))
        tc.copy_(torch.from_numpy(cxy * scale))
        torch.cuda.synchronize()
        g.launch()
        torch.cuda.synchronize()
        got = [x.cpu().numpy() for x in out]
        if scale == 1.0:
            assert same(first, got)
    g.close()
    assert same(separate(), got)

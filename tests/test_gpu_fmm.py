"""GPU parity tests: the CUDA library through its C ABI against the oracle.

Bars (stated per check):
* tree, keys, body order, M2L/P2P list sets: bit-exact;
* FP64 expansions and results: relative error <= 1e-11 (different summation
  order and libm vs CUDA math, both FP64);
* mixed form: rel-L2 vs the FP64 form <= 2e-6, and vs direct sum the same
  accuracy class as FP64.
"""
import contextlib
import pathlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = sorted(p for p in (pathlib.Path(__file__).parent / "golden").glob("*.npz")
                if not p.stem.startswith(("bh_", "refsample_", "io_")))
FP64_RTOL = 1e-11


def _cells_by_key(c, key_name="key"):
    order = np.argsort(c[key_name], kind="stable")
    return order


def _rel(a, b):
    scale = max(np.max(np.abs(b)), 1e-300)
    return float(np.max(np.abs(a - b)) / scale)


def _rel_rows(a, b):
    """max over rows of |a-b| / |b| (row norms), for per-body 4-vectors."""
    num = np.linalg.norm(a - b, axis=-1)
    den = np.maximum(np.linalg.norm(b, axis=-1), 1e-300)
    return float(np.max(num / den))


CASES = [
    ("uniform_cube", 20000, 1, 10, 64, 0.4),
    ("plummer", 30000, 2, 8, 32, 0.5),
    ("sphere_surface", 25000, 5, 6, 16, 0.35),
    ("two_gaussians", 15000, 4, 12, 128, 0.3),
    ("uniform_cube", 3000, 7, 4, 1, 0.6),
]
IDS = [f"{c[0]}-n{c[1]}-p{c[3]}-ncrit{c[4]}" for c in CASES]


@pytest.fixture(scope="module", params=CASES, ids=IDS)
def run(request, tb, oracle_mod, ctx):
    dist, n, seed, P, ncrit, theta = request.param
    x, y, z, q = tb.datasets.make(dist, n, seed)
    o = oracle_mod.Oracle(x, y, z, q, P=P, ncrit=ncrit, theta=theta)
    ctx.partition(x, y, z, q, ncrit=ncrit)
    ctx.upward(P, tb.FP64)
    # lists exactly as the reference's traversal visits them ...
    ctx.set_reference_lists(True)
    ctx.build_lists(theta)
    lists = ctx.lists()
    linfo = ctx.list_info()
    # ... and the default lists without pairs of empty cells, used for the results
    ctx.set_reference_lists(False)
    ctx.build_lists(theta)
    pruned = ctx.lists()
    ctx.m2l(tb.FP64)
    ctx.p2p(tb.FP64)
    ctx.downward(tb.FP64)
    res = ctx.results(tb.ORDER_ORIGINAL)
    cells = ctx.cells()
    sorted_idx, sorted_keys = ctx.sorted_bodies()
    M, L = ctx.expansions()
    return dict(x=x, y=y, z=z, q=q, P=P, theta=theta, o=o, res=res, cells=cells, lists=lists,
                sorted_idx=sorted_idx, sorted_keys=sorted_keys, M=M, L=L,
                info=ctx.tree_info(), linfo=linfo, pruned=pruned)


def test_tree_bit_exact(run):
    o = run["o"]
    oi, ok, _ = o.bodies()
    assert np.array_equal(run["sorted_keys"], ok)
    assert np.array_equal(run["sorted_idx"], oi)
    oc = o.cells()
    gc = run["cells"]
    assert len(gc["key"]) == len(oc["key"])
    go, oo = _cells_by_key(gc), _cells_by_key(oc)
    assert np.array_equal(gc["key"][go], oc["key"][oo])
    assert np.array_equal(gc["leaf"][go], oc["leaf"][oo])
    assert np.array_equal(gc["nb"][go], oc["nb"][oo])
    assert np.array_equal(gc["bbeg"][go].astype(np.int64), oc["bid"][oo])
    assert np.array_equal(gc["center"][go], oc["center"][oo])
    assert np.array_equal(gc["width"][go], oc["width"][oo])
    lo_hi = o.bbox()
    assert run["info"]["box_lo"] == lo_hi[0] and run["info"]["box_hi"] == lo_hi[1]


def _pair_keys(keys, t, s):
    return set(zip(keys[t].tolist(), keys[s].tolist()))


def test_lists_equal_as_sets(run):
    o = run["o"]
    okeys = o.cells()["key"]
    gkeys = run["cells"]["key"]
    (gmt, gms), (gpt, gps) = run["lists"]
    omt, oms = o.m2l_list()
    opt, ops = o.p2p_list()
    assert len(gmt) == len(omt) and len(gpt) == len(opt)
    assert _pair_keys(gkeys, gmt, gms) == _pair_keys(okeys, omt, oms)
    assert _pair_keys(gkeys, gpt, gps) == _pair_keys(okeys, opt, ops)
    assert run["linfo"]["n_p2p_interactions"] == o.p2p_interactions()
    # sorted by (target, source)
    packed = gmt.astype(np.int64) * (1 << 32) + gms
    assert np.all(np.diff(packed) > 0)


def test_pruned_lists_drop_only_empty_pairs(run):
    """Default lists = reference lists minus the pairs with an empty cell."""
    gkeys, nb = run["cells"]["key"], run["cells"]["nb"]
    (rmt, rms), (rpt, rps) = run["lists"]
    (pmt, pms), (ppt, pps) = run["pruned"]
    keep = (nb[rmt] > 0) & (nb[rms] > 0)
    assert _pair_keys(gkeys, pmt, pms) == _pair_keys(gkeys, rmt[keep], rms[keep])
    assert _pair_keys(gkeys, ppt, pps) == _pair_keys(gkeys, rpt, rps)


def test_expansions_fp64(run):
    o = run["o"]
    oM, oL = o.expansions()
    oc, gc = o.cells(), run["cells"]
    go, oo = _cells_by_key(gc), _cells_by_key(oc)
    assert _rel(run["M"][go], oM[oo]) < FP64_RTOL
    # L of empty cells is never used (and not computed on the GPU).
    ne = oc["nb"][oo] > 0
    assert _rel(run["L"][go][ne], oL[oo][ne]) < FP64_RTOL


def test_results_fp64(run):
    ref = run["o"].result()
    res = run["res"]
    assert _rel(res[:, 0], ref[:, 0]) < FP64_RTOL
    assert _rel(res[:, 1:], ref[:, 1:]) < FP64_RTOL
    assert _rel_rows(res, ref) < 1e-9


@pytest.mark.parametrize("path", GOLDEN, ids=[p.stem for p in GOLDEN])
def test_against_reference_goldens(path, tb, ctx):
    """Directly against outputs of the unmodified reference (with the golden's
    mutual option: the example's -m)."""
    g = np.load(path)
    mutual = int(g["mutual"]) if "mutual" in g else 0
    ctx.set_reference_lists(True)
    try:
        ctx.partition(g["x"], g["y"], g["z"], g["q"], ncrit=int(g["ncrit"]))
        ctx.upward(int(g["P"]), tb.FP64)
        ctx.traverse(float(g["theta"]), mutual, tb.FP64)
        ctx.downward(tb.FP64)
        res = ctx.results(tb.ORDER_ORIGINAL)
    finally:
        ctx.set_reference_lists(False)
    c = ctx.cells()
    order = np.argsort(c["key"], kind="stable")
    assert np.array_equal(c["key"][order], g["cell_key"])
    assert np.array_equal(c["nb"][order], g["cell_nb"])
    assert np.array_equal(c["leaf"][order], g["cell_leaf"])
    li = ctx.list_info()
    if mutual:
        # the lists hold both directions of every unordered pair the reference
        # visited; its counters count visits (j <= i within a leaf)
        (mt, ms), (pt, ps) = ctx.lists()
        nb = c["nb"].astype(np.int64)
        up = pt < ps
        self_ = pt == ps
        visits = int(np.sum(nb[pt[up]] * nb[ps[up]]) +
                     np.sum(nb[pt[self_]] * (nb[pt[self_]] + 1) // 2))
        assert li["n_m2l"] == 2 * int(g["n_m2l"])
        assert visits == int(g["n_p2p_interactions"])
    else:
        assert li["n_m2l"] == int(g["n_m2l"])
        assert li["n_p2p_interactions"] == int(g["n_p2p_interactions"])
    assert _rel(res, g["trg"]) < FP64_RTOL
    if "M" in g:
        M, L = ctx.expansions()
        assert _rel(M[order], g["M"]) < FP64_RTOL
        ne = g["cell_nb"] > 0
        assert _rel(L[order][ne], g["L"][ne]) < FP64_RTOL


@pytest.mark.parametrize("dist,ncrit", [("plummer", 64), ("plummer", 16),
                                        ("sphere_surface", 128), ("uniform_cube", 128)])
def test_mixed_close_to_fp64(dist, ncrit, tb, ctx, oracle_mod):
    """Mixed near field and tensor-core M2L against the FP64 form: small
    leaves (4-target P2P tiles) and full leaves (3-target tiles at 16 warps)."""
    x, y, z, q = tb.datasets.make(dist, 40000, 21)
    r64 = ctx.evaluate(x, y, z, q, P=10, ncrit=ncrit, theta=0.4, precision=tb.FP64)
    rmx = ctx.evaluate(x, y, z, q, P=10, ncrit=ncrit, theta=0.4, precision=tb.MIXED)
    ep, ea = oracle_mod.rel_l2(rmx, r64)
    assert ep < 2e-6 and ea < 2e-6
    tg = tb.datasets.sample_targets(len(x), 500)
    d = ctx.direct(tg)
    e64 = oracle_mod.rel_l2(r64[tg], d)
    emx = oracle_mod.rel_l2(rmx[tg], d)
    assert emx[0] < 1.5 * e64[0] + 1e-6 and emx[1] < 1.5 * e64[1] + 1e-6


@pytest.mark.parametrize("P", [14, 16])
def test_mixed_high_order_deep_tree(P, tb, ctx, oracle_mod):
    """Mixed form at high order on a deep tree: in small cells the local
    coefficients of degree n grow like 1/R^(n+1), beyond the FP32 range, so
    the FP32 L2P must work in units of the leaf width.  The results are finite
    and within 2e-6 (rel-L2) of the FP64 form."""
    x, y, z, q = tb.datasets.make("two_gaussians", 200000, 7)
    r64 = ctx.evaluate(x, y, z, q, P=P, ncrit=32, theta=0.4, precision=tb.FP64)
    rmx = ctx.evaluate(x, y, z, q, P=P, ncrit=32, theta=0.4, precision=tb.MIXED)
    assert np.isfinite(rmx).all()
    ep, ea = oracle_mod.rel_l2(rmx, r64)
    assert ep < 2e-6 and ea < 2e-6


@pytest.mark.parametrize("P", [4, 6, 8, 10, 11, 12, 14, 16])
def test_tensorcore_m2l_matches_fp64(P, tb, ctx):
    """Split-TF32 tensor-core M2L (mixed) against the FP64 M2L: per cell,
    ||L_mixed - L_fp64|| / ||L_fp64|| <= 2e-5 (FP32 accumulation of ~100-300
    translations of ~1e-7 relative accuracy each)."""
    x, y, z, q = tb.datasets.make("plummer", 60000, 61)
    ctx.partition(x, y, z, q, ncrit=32)
    ctx.upward(P, tb.FP64)
    ctx.build_lists(0.4)
    ctx.m2l(tb.FP64)
    _, L64 = ctx.expansions()
    ctx.m2l(tb.MIXED)
    _, Lmx = ctx.expansions()
    nb = ctx.cells()["nb"]
    ne = (nb > 0) & (np.linalg.norm(L64, axis=1) > 0)
    rel = np.linalg.norm(Lmx[ne] - L64[ne], axis=1) / np.linalg.norm(L64[ne], axis=1)
    assert rel.max() < 2e-5, (rel.max(), np.median(rel))


def test_gpu_direct_matches_oracle_direct(tb, ctx, oracle_mod):
    x, y, z, q = tb.datasets.make("uniform_cube", 20000, 3)
    ctx.partition(x, y, z, q, ncrit=64)
    tg = tb.datasets.sample_targets(len(x), 64)
    d = ctx.direct(tg)
    ref = oracle_mod.direct(x, y, z, q, tg, field=True)
    assert _rel(d, ref) < 1e-12


def test_fp64_accuracy_vs_direct(tb, ctx, oracle_mod):
    # The reference's own accuracy gate is rel-L2 < 5e-3 (test.sh:234); at
    # P=10, theta=0.4 the method gives ~1e-5 on zero-mean-free data.
    x, y, z, q = tb.datasets.make("uniform_cube", 50000, 9)
    r = ctx.evaluate(x, y, z, q, P=10, ncrit=64, theta=0.4, precision=tb.FP64)
    tg = tb.datasets.sample_targets(len(x), 300)
    ep, ea = oracle_mod.rel_l2(r[tg], ctx.direct(tg))
    assert ep < 1e-4 and ea < 1e-3


def test_deterministic(tb, ctx):
    """The FP64 form is bit-reproducible (lists sorted, no atomics).  The mixed
    form adds tensor-core M2L columns into FP32 locals with atomic reductions,
    so the summation order, and the last bits, vary between runs: repeat runs
    agree to 1e-7 relative."""
    x, y, z, q = tb.datasets.make("plummer", 30000, 23)
    a = ctx.evaluate(x, y, z, q, P=8, ncrit=32, theta=0.4, precision=tb.FP64)
    b = ctx.evaluate(x, y, z, q, P=8, ncrit=32, theta=0.4, precision=tb.FP64)
    assert np.array_equal(a, b)
    a = ctx.evaluate(x, y, z, q, P=8, ncrit=32, theta=0.4, precision=tb.MIXED)
    b = ctx.evaluate(x, y, z, q, P=8, ncrit=32, theta=0.4, precision=tb.MIXED)
    assert _rel(a, b) < 1e-7


def test_class_key_ranges_reused_and_renewed(tb, ctx):
    """The M2L class keys are packed with the field ranges of the previous
    classification; a list with larger offsets (smaller theta) misses them and
    is classified again.  Either way the classes, and so the FP64 class-GEMM
    result, equal a fresh context's bit for bit."""
    x, y, z, q = tb.datasets.make("plummer", 60000, 41)
    fresh = tb.Context(0)
    try:
        ref = {th: fresh.evaluate(x, y, z, q, P=8, ncrit=32, theta=th, precision=tb.FP64)
               for th in (0.3, 0.6)}
    finally:
        fresh.close()
    for th in (0.6, 0.3, 0.3, 0.6):
        r = ctx.evaluate(x, y, z, q, P=8, ncrit=32, theta=th, precision=tb.FP64)
        assert np.array_equal(r, ref[th])


def test_mixed_traverse_lists_sorted_on_demand(tb, ctx):
    """The mixed form's traversal leaves each target's sources unsorted in both
    lists (its M2L regroups the pairs by offset class, its FP32 near field sums
    in any order); the list accessor and a later FP64 M2L and P2P see them
    sorted, as build_lists gives them, so an FP64 evaluation after a mixed
    traversal equals a plain one bit for bit."""
    x, y, z, q = tb.datasets.make("sphere_surface", 40000, 3)
    fp64 = ctx.evaluate(x, y, z, q, P=6, ncrit=32, theta=0.4, precision=tb.FP64)
    (mt0, ms0), (pt0, ps0) = ctx.lists()
    ctx.upward(P=6, precision=tb.FP64)
    ctx.traverse(0.4, 0, tb.MIXED)
    (mt, ms), (pt, ps) = ctx.lists()
    for a, b in ((mt, mt0), (ms, ms0), (pt, pt0), (ps, ps0)):
        assert np.array_equal(a, b)
    assert np.all(np.diff(mt.astype(np.int64) * (1 << 32) + ms) > 0)
    ctx.traverse(0.4, 0, tb.MIXED)
    ctx.m2l(tb.FP64)
    ctx.p2p(tb.FP64)
    ctx.downward(tb.FP64)
    assert np.array_equal(ctx.results(), fp64)


@pytest.mark.parametrize("n,ncrit", [(1, 64), (2, 1), (5, 2), (50, 64), (64, 64), (65, 64)])
def test_small_and_root_leaf(n, ncrit, tb, ctx, oracle_mod):
    """Tiny inputs, including a root that is itself a leaf (which the reference
    itself cannot run) and the bounding-cube quirk with few bodies."""
    x, y, z, q = tb.datasets.make("uniform_cube", n, 31 + n)
    o = oracle_mod.Oracle(x, y, z, q, P=6, ncrit=ncrit, theta=0.4)
    r = ctx.evaluate(x, y, z, q, P=6, ncrit=ncrit, theta=0.4, precision=tb.FP64)
    ref = o.result()
    assert np.array_equal(np.isnan(r), np.isnan(ref))
    ok = ~np.isnan(ref)
    if ok.any():
        assert _rel(r[ok], ref[ok]) < FP64_RTOL
    gi, gk = ctx.sorted_bodies()
    oi, ok2, _ = o.bodies()
    assert np.array_equal(gk, ok2) and np.array_equal(gi, oi)


def test_coincident_bodies_reach_max_depth(tb, ctx, oracle_mod):
    """More than ncrit bodies at one point: cells split to the deepest key
    level (19), where they become leaves."""
    x, y, z, q = [a.copy() for a in tb.datasets.make("uniform_cube", 400, 41)]
    x[:40] = 0.123
    y[:40] = -0.456
    z[:40] = 0.789
    o = oracle_mod.Oracle(x, y, z, q, P=4, ncrit=8, theta=0.5)
    r = ctx.evaluate(x, y, z, q, P=4, ncrit=8, theta=0.5, precision=tb.FP64)
    assert ctx.tree_info()["max_depth"] == 19
    ref = o.result()
    assert _rel(r, ref) < FP64_RTOL


def test_errors_are_status_codes(tb):
    with tb.Context(0) as c:
        with pytest.raises(tb.TapasError) as e:
            c.upward(10)
        assert e.value.code == -4  # state: no tree
        x, y, z, q = tb.datasets.make("uniform_cube", 1000, 1)
        c.partition(x, y, z, q, ncrit=16)
        with pytest.raises(tb.TapasError) as e:
            c.upward(17)
        assert e.value.code == -6
        c.upward(6)
        with pytest.raises(tb.TapasError) as e:
            c.build_lists(0.4, mutual=2)
        assert e.value.code == -1
        with pytest.raises(tb.TapasError) as e:
            c.downward()
        assert e.value.code == -4
        with pytest.raises(tb.TapasError) as e:
            c.partition(x, y, z, q, ncrit=0)
        assert e.value.code == -1


def test_device_pointers(tb, ctx):
    torch = pytest.importorskip("torch")
    x, y, z, q = tb.datasets.make("uniform_cube", 10000, 51)
    ref = ctx.evaluate(x, y, z, q, P=6, ncrit=32, theta=0.4)
    dx, dy, dz, dq = [torch.from_numpy(a).cuda() for a in (x, y, z, q)]
    out = torch.zeros((len(x), 4), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.evaluate(dx, dy, dz, dq, P=6, ncrit=32, theta=0.4, out=out)
    assert np.array_equal(out.cpu().numpy(), ref)


@pytest.mark.parametrize("ncrit,nsparse,longest", [(64, 120, 4000), (8, 16, 30000)],
                         ids=["block-sorted", "radix-sorted"])
def test_long_list_segments(tb, oracle_mod, ctx, ncrit, nsparse, longest):
    """Leaves of a sparse half-cube beside a dense half each have a P2P list of
    thousands of small leaves: longer than one warp sorts (a block sorts
    them), or longer than one block sorts (the whole list goes through the
    radix sort).  Both lists must still equal the reference traversal's as
    sets, in (target, source) order."""
    rng = np.random.default_rng(11)
    dense = rng.random((120000, 3))
    dense[:, 0] *= 0.5
    sparse = rng.random((nsparse, 3))
    sparse[:, 0] = 0.5 + 0.5 * sparse[:, 0]
    pts = np.vstack([dense, sparse])
    x, y, z = (np.ascontiguousarray(pts[:, d]) for d in range(3))
    q = rng.random(len(x)) / len(x)
    o = oracle_mod.Oracle(x, y, z, q, P=4, ncrit=ncrit, theta=0.3, run=False)
    assert oracle_mod.lib().oracle_build(o.h) == 0
    assert oracle_mod.lib().oracle_traverse(o.h) == 0
    ctx.partition(x, y, z, q, ncrit=ncrit)
    ctx.set_reference_lists(True)
    try:
        ctx.build_lists(0.3)
        (gmt, gms), (gpt, gps) = ctx.lists()
    finally:
        ctx.set_reference_lists(False)
    assert np.bincount(gpt).max() > longest  # the path is exercised
    gkeys, okeys = ctx.cells()["key"], o.cells()["key"]
    omt, oms = o.m2l_list()
    opt, ops = o.p2p_list()
    assert _pair_keys(gkeys, gmt, gms) == _pair_keys(okeys, omt, oms)
    assert _pair_keys(gkeys, gpt, gps) == _pair_keys(okeys, opt, ops)
    for t, s in ((gmt, gms), (gpt, gps)):
        assert np.all(np.diff(t.astype(np.int64) * (1 << 32) + s) > 0)


def test_long_source_lists_are_split(tb, ctx):
    """A Plummer set has leaves whose near-field lists hold far more than the
    32,768 source bodies one P2P work item takes; those lists are cut into
    pieces whose partial sums are added in piece order, so the FP64 form stays
    bit-reproducible and both forms keep their accuracy."""
    x, y, z, q = tb.datasets.make("plummer", 200000, 31)
    ctx.partition(x, y, z, q, ncrit=64)
    ctx.build_lists(0.3)
    c = ctx.cells()
    _, (pt, ps) = ctx.lists()
    per_target = np.bincount(pt, weights=c["nb"][ps].astype(np.float64), minlength=len(c["nb"]))
    assert per_target.max() > 4 * 32768  # the case is exercised
    a = ctx.evaluate(x, y, z, q, P=8, ncrit=64, theta=0.3, precision=tb.FP64)
    b = ctx.evaluate(x, y, z, q, P=8, ncrit=64, theta=0.3, precision=tb.FP64)
    assert np.array_equal(a, b)
    tg = tb.datasets.sample_targets(len(x), 400, seed=5)
    d = ctx.direct(tg)
    num = np.linalg.norm(a[tg] - d, axis=0)
    den = np.linalg.norm(d, axis=0)
    assert num[0] / den[0] < 1e-5 and np.linalg.norm(num[1:]) / np.linalg.norm(den[1:]) < 1e-4
    m = ctx.evaluate(x, y, z, q, P=8, ncrit=64, theta=0.3, precision=tb.MIXED)
    assert np.linalg.norm(m[:, 0] - a[:, 0]) / np.linalg.norm(a[:, 0]) < 2e-6


def test_tensorcore_m2l_wait_timeout_is_a_status(tb, ctx):
    """The tensor-core M2L's designed failure path: with a wait bound of 100
    clock cycles the MMA thread's first wait for a copy gives up, every role
    leaves its loop, the CTA drains its copies and MMAs and frees its tensor
    memory, and the call returns TAPAS_B200_ERR_TIMEOUT.  The same context then
    evaluates normally with the default bound."""
    x, y, z, q = tb.datasets.make("plummer", 60000, 61)
    ctx.partition(x, y, z, q, ncrit=32)
    ctx.upward(8, tb.FP64)
    ctx.build_lists(0.4)
    ctx.m2l(tb.FP64)
    _, L64 = ctx.expansions()
    try:
        ctx.set_wait_limit(100)
        with pytest.raises(tb.TapasError) as e:
            ctx.m2l(tb.MIXED)
        assert e.value.code == tb._lib.ERR_TIMEOUT
        assert "gave up" in str(e.value)
    finally:
        ctx.set_wait_limit(0)
    ctx.m2l(tb.MIXED)
    _, Lmx = ctx.expansions()
    nb = ctx.cells()["nb"]
    ne = (nb > 0) & (np.linalg.norm(L64, axis=1) > 0)
    rel = np.linalg.norm(Lmx[ne] - L64[ne], axis=1) / np.linalg.norm(L64[ne], axis=1)
    assert rel.max() < 2e-5


@pytest.mark.parametrize("P", [6, 12, 16])
def test_mixed_tree_translations_per_cell(P, tb, ctx):
    """The mixed form's tree translations (M2M: split-TF32 tensor-core GEMMs
    with level-independent operators on the deepest three parent levels below
    level 3, FP64 level GEMMs above them; L2L: FP64) on a deep tree, per cell
    against the FP64 form: multipoles within 1e-6 of
    the cell's multipoles of |q| (see below), local expansions after the
    downward pass within 5e-5 of the FP64 ones."""
    x, y, z, q = tb.datasets.make("two_gaussians", 200000, 19)
    ctx.partition(x, y, z, np.abs(q), ncrit=32)
    ctx.upward(P, tb.FP64)
    Mabs, _ = ctx.expansions()
    assert ctx.tree_info()["max_depth"] >= 8  # levels below the FP64 ones exist
    out = {}
    for prec in (tb.FP64, tb.MIXED):
        ctx.partition(x, y, z, q, ncrit=32)
        ctx.upward(P, prec)
        ctx.traverse(0.4, 0, prec)
        ctx.downward(prec)
        out[prec] = ctx.expansions()
    (M64, L64), (Mmx, Lmx) = out[tb.FP64], out[tb.MIXED]
    scale = np.linalg.norm(Mabs, axis=1)
    ok = scale > 0
    relM = np.linalg.norm(Mmx[ok] - M64[ok], axis=1) / scale[ok]
    assert relM.max() < 1e-6, relM.max()
    nrm = np.linalg.norm(L64, axis=1)
    ne = (ctx.cells()["nb"] > 0) & (nrm > 0)
    relL = np.linalg.norm(Lmx[ne] - L64[ne], axis=1) / nrm[ne]
    assert relL.max() < 5e-5, (relL.max(), np.median(relL))


@pytest.mark.parametrize("P", [4, 10, 16])
@pytest.mark.parametrize("dist", ["sphere_surface", "two_gaussians"])
def test_fp32_p2m_per_cell(P, dist, tb, ctx):
    """The mixed form's P2M (FP32 terms in units of the leaf width, FP32 warp
    reduce-scatter, FP64 sums over body chunks) followed by its M2M (FP64 at
    the top levels, split-TF32 tensor cores below), against the FP64 upward
    pass, per cell.  An FP32 term rounds to ~6e-8 of
    itself, so the error of a cell's M is bounded by its scale without
    cancellation: ||M_mixed - M_fp64|| <= 1e-6 ||M_|q|||, M_|q| the FP64
    multipoles of the charges' magnitudes.  (Where zero-mean charges cancel,
    M_fp64 itself can be far smaller than that scale.)  The sphere-surface set
    has zero-mean charges; the Gaussian clusters give a deep tree."""
    x, y, z, q = tb.datasets.make(dist, 150000, 17)
    ctx.partition(x, y, z, np.abs(q), ncrit=32)
    ctx.upward(P, tb.FP64)
    Mabs, _ = ctx.expansions()
    ctx.partition(x, y, z, q, ncrit=32)
    ctx.upward(P, tb.FP64)
    M64, _ = ctx.expansions()
    ctx.upward(P, tb.MIXED)
    Mmx, _ = ctx.expansions()
    scale = np.linalg.norm(Mabs, axis=1)
    ok = scale > 0
    rel = np.linalg.norm(Mmx[ok] - M64[ok], axis=1) / scale[ok]
    assert rel.max() < 1e-6, (rel.max(), np.median(rel))
    assert ctx.tree_info()["max_depth"] >= 6


@pytest.mark.parametrize("P", [4, 5, 7, 9, 11, 13, 15, 16])
def test_fp64_m2l_products_every_order(P, tb, ctx, oracle_mod):
    """The FP64 M2L's class products (32-pair, 32-output, 16-source blocks:
    every order ends differently) and its rare classes' pairs against the
    oracle's L, with the reference's lists (pairs of empty cells have no product
    row) and without them.  Same bar as the other FP64 expansions."""
    x, y, z, q = tb.datasets.make("two_gaussians", 1500, 19)
    o = oracle_mod.Oracle(x, y, z, q, P=P, ncrit=8, theta=0.45)
    _, oL = o.expansions()
    oc = o.cells()
    oo = _cells_by_key(oc)
    ne = oc["nb"][oo] > 0
    ctx.partition(x, y, z, q, ncrit=8)
    ctx.upward(P, tb.FP64)
    Ls = []
    for keep in (True, False):
        ctx.set_reference_lists(keep)
        ctx.build_lists(0.45)
        ctx.set_reference_lists(False)
        ctx.m2l(tb.FP64)
        ctx.p2p(tb.FP64)
        ctx.downward(tb.FP64)
        Ls.append(ctx.expansions()[1])
    go = _cells_by_key(ctx.cells())
    assert _rel(Ls[0][go][ne], oL[oo][ne]) < FP64_RTOL
    assert _rel(Ls[1][go][ne], oL[oo][ne]) < FP64_RTOL


def test_fp64_m2l_rows_in_ranges(tb, ctx, oracle_mod):
    """A list whose product rows exceed the buffer (512 MiB: 247k pairs at P = 16)
    is evaluated in ranges that cut targets; a pair left out or added twice
    would show at the 1e-3 level, the truncation error of P = 16, theta = 0.3
    on this workload is below 1e-5."""
    x, y, z, q = tb.datasets.make("uniform_cube", 60000, 12)
    a = ctx.evaluate(x, y, z, q, P=16, ncrit=16, theta=0.3, precision=tb.FP64)
    assert ctx.list_info()["n_m2l"] > 2 * 987000
    tg = tb.datasets.sample_targets(len(x), 300)
    ep, ea = oracle_mod.rel_l2(a[tg], ctx.direct(tg))
    assert ep < 1e-5 and ea < 1e-5
    b = ctx.evaluate(x, y, z, q, P=16, ncrit=16, theta=0.3, precision=tb.FP64)
    assert np.array_equal(a, b)


@pytest.mark.parametrize("n,k", [(1, 1), (7, 3), (127, 8), (129, 9), (5000, 17), (40001, 1)])
def test_direct_tile_edges(n, k, tb, ctx, oracle_mod):
    """Part-filled target tiles, few sources, coincident bodies; the no-alloc
    form over the same tiles.  Bar as the other direct-sum test."""
    x, y, z, q = [a.copy() for a in tb.datasets.make("uniform_cube", n, 5)]
    if n > 6:
        x[1], y[1], z[1] = x[0], y[0], z[0]  # coincident: their pair adds nothing
        x[3] = x[2] + 1e-9
        y[3], z[3] = y[2], z[2]
    ctx.partition(x, y, z, q, ncrit=64)
    tg = (np.arange(k) * 7919) % n
    d = ctx.direct(tg)
    ref = oracle_mod.direct(x, y, z, q, tg, field=True)
    assert _rel(d, ref) < 1e-12
    import torch
    dev = [torch.from_numpy(a).cuda() for a in (x, y, z, q)]
    t = torch.from_numpy(tg.astype(np.int64)).cuda()
    out = torch.zeros((k, 4), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert tb.lib().tapas_b200_direct_noalloc(*[a.data_ptr() for a in dev], n, t.data_ptr(), k,
                                              out.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert _rel(out.cpu().numpy(), ref) < 1e-12


@pytest.mark.parametrize("n,ncrit", [(40, 1), (900, 2), (1500, 9), (3000, 40), (2500, 150),
                                     (3000, 300), (290, 300), (12000, 600)])
def test_near_field_tile_shapes(n, ncrit, tb, ctx, oracle_mod):
    """Leaves of one body up to several hundred: every tile shape (1, 3 or 4
    targets per lane, sources split over up to 32 lane groups), leaves of more
    than one tile (128 targets), target lists long enough to be split into
    pieces, coincident and nearly coincident bodies.  FP64 against the oracle,
    mixed against FP64, at their bars."""
    x, y, z, q = [a.copy() for a in tb.datasets.make("two_gaussians", n, 57)]
    x[1], y[1], z[1] = x[0], y[0], z[0]
    x[3] = x[2] + 1e-6
    y[3], z[3] = y[2], z[2]
    ref = oracle_mod.Oracle(x, y, z, q, P=6, ncrit=ncrit, theta=0.3).result()
    r64 = ctx.evaluate(x, y, z, q, P=6, ncrit=ncrit, theta=0.3, precision=tb.FP64)
    assert _rel(r64[:, 0], ref[:, 0]) < FP64_RTOL
    assert _rel(r64[:, 1:], ref[:, 1:]) < FP64_RTOL
    rmx = ctx.evaluate(x, y, z, q, P=6, ncrit=ncrit, theta=0.3, precision=tb.MIXED)
    ep, ea = oracle_mod.rel_l2(rmx, r64)
    assert ep < 2e-6 and ea < 2e-6


def _check_tree(tb, ctx, oracle_mod, x, y, z, q, ncrit):
    o = oracle_mod.Oracle(x, y, z, q, P=2, ncrit=ncrit, theta=5.0)
    info = ctx.partition(x, y, z, q, ncrit=ncrit)
    oi, ok, _ = o.bodies()
    gi, gk = ctx.sorted_bodies()
    assert np.array_equal(gk, ok)
    assert np.array_equal(gi, oi)
    oc, gc = o.cells(), ctx.cells()
    go, oo = _cells_by_key(gc), _cells_by_key(oc)
    for name, ours in (("key", "key"), ("leaf", "leaf"), ("nb", "nb"), ("center", "center"),
                       ("width", "width")):
        assert np.array_equal(gc[ours][go], oc[name][oo]), name
    assert np.array_equal(gc["bbeg"][go].astype(np.int64), oc["bid"][oo])
    # breadth first, children after their parent, eight in a row
    assert info["n_cells"] == len(gc["key"])
    level = gc["key"] & np.uint64(31)
    assert np.all(np.diff(level.astype(np.int64)) >= 0)
    inner = np.flatnonzero(gc["leaf"] == 0)
    for k in range(8):
        assert np.array_equal(gc["parent"][gc["child0"][inner] + k], inner)
    assert np.all(gc["child0"][gc["leaf"] != 0] == -1)


@pytest.mark.parametrize("n,ncrit", [(2047, 1), (2048, 7), (2049, 300), (4096, 1), (4097, 2),
                                     (6145, 16), (33, 32), (300, 299)])
def test_tree_all_levels_at_once(n, ncrit, tb, ctx, oracle_mod):
    """Body counts around the counting pass's warps and blocks and the one-block
    sort's limit, few and many levels, against the oracle's tree, bit for bit."""
    x, y, z, q = tb.datasets.make("two_gaussians" if n % 2 else "uniform_cube", n, 91)
    _check_tree(tb, ctx, oracle_mod, x, y, z, q, ncrit)


@pytest.mark.parametrize("n", [1500, 9000])
@pytest.mark.parametrize("longest", [3, 31, 33])
def test_tree_bodies_close_in_one_cell(n, longest, tb, ctx, oracle_mod):
    """Clusters far smaller than a cell of level 13: the sort orders runs of up to
    32 such bodies after its high key bits and starts over on all bits for a
    longer one; some bodies coincide (equal keys stay in input order)."""
    x, y, z, q = [a.copy() for a in tb.datasets.make("uniform_cube", n, 92)]
    rng = np.random.default_rng(5)
    for k, at in enumerate(range(0, n - longest, n // 7)):
        m = longest if k == 3 else 1 + k % 3
        idx = rng.permutation(n)[:m]
        for a, c in ((x, 0.3), (y, -0.2), (z, 0.6)):
            a[idx] = c + 0.1 * k + 3e-6 * rng.random(m)
        if m > 1:
            x[idx[1]], y[idx[1]], z[idx[1]] = x[idx[0]], y[idx[0]], z[idx[0]]
    _check_tree(tb, ctx, oracle_mod, x, y, z, q, 4)


@pytest.mark.parametrize("n", [1, 700, 30000])
def test_near_field_counts_belong_to_their_call(n, tb, ctx):
    """traverse() counts the near field's work ahead of the M2L; a p2p() call after
    it, at the other precision or after new lists, counts its own: bit for bit the
    result of a p2p() with nothing before it."""
    b = tb.datasets.make("two_gaussians", n, 61)

    def alone(theta, precision, before):
        ctx.partition(*b, ncrit=16)
        ctx.upward(4, tb.MIXED)
        if before:
            ctx.traverse(0.5, precision=tb.MIXED)
        if theta is not None:
            ctx.build_lists(theta)
        ctx.p2p(precision)
        return ctx.results()

    for precision in (tb.FP64, tb.MIXED):
        assert np.array_equal(alone(0.5, precision, False), alone(None, precision, True))
        assert np.array_equal(alone(0.8, precision, False), alone(0.8, precision, True))


@pytest.mark.parametrize("P,exponent", [(16, 66), (16, 40), (10, 101), (10, -95)])
def test_fp64_evaluation_in_other_units(P, exponent, tb, ctx):
    """Bodies in units so small or large that the powers of a cell's width leave the
    FP64 range (cells of 2^64 and more at P = 16, as a galaxy's in metres): scaled by a
    power of two the evaluation is the same up to the local coefficients that
    become subnormal; those of degree 15 carry ~1e-6 of the field and keep 18 bits."""
    x, y, z, q = tb.datasets.make("uniform_cube", 3000, 12)
    args = dict(P=P, ncrit=16, theta=0.4, precision=tb.FP64)
    a = ctx.evaluate(x, y, z, q, **args)
    s = 2.0 ** exponent
    b = ctx.evaluate(x * s, y * s, z * s, q, **args) * np.array([s, s * s, s * s, s * s])
    assert np.isfinite(b).all()
    assert _rel(b[:, 0], a[:, 0]) < 1e-8 and _rel(b[:, 1:], a[:, 1:]) < 1e-8


def test_mixed_evaluation_after_a_zero_width_tree(tb):
    """Bodies all at one point make a deep tree of zero-width cells; what a context
    keeps from it (the M2M operators belong to an order, not to a tree) leaves the
    next evaluation as in a context of its own."""
    b = tb.datasets.make("plummer", 30000, 3)
    point, ones = np.full(60, 0.25), np.ones(60)
    args = dict(P=8, ncrit=8, theta=0.4, precision=tb.MIXED)
    with tb.Context(0) as c:
        ref = c.evaluate(*b, **args)
    with tb.Context(0) as c:
        c.evaluate(point, point, point, ones, **args)
        got = c.evaluate(*b, **args)
    assert np.isfinite(got).all()
    # the mixed form's FP32 reductions are added in no fixed order
    assert np.linalg.norm(got - ref, axis=0).max() <= 1e-6 * np.linalg.norm(ref, axis=0).max()


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_set_multipoles_after_upward(precision, tb, ctx):
    """Multipoles given after a whole upward pass are the ones the M2L translates:
    doubled, the local expansions double (exactly, but for the mixed form's FP32
    reductions in no fixed order)."""
    x, y, z, q = tb.datasets.make("uniform_cube", 20000, 3)
    ctx.partition(x, y, z, q, ncrit=64)
    ctx.upward(8, precision)
    ctx.build_lists(0.4)
    M = ctx.multipoles()
    ctx.m2l(precision)
    L1 = ctx.expansions()[1]
    ctx.set_multipoles(np.stack([2 * M.real, 2 * M.imag], axis=-1))
    ctx.m2l(precision)
    L2 = ctx.expansions()[1]
    ne = ctx.cells()["nb"] > 0
    tol = 0.0 if precision == tb.FP64 else 1e-6
    assert np.linalg.norm(L2[ne] - 2 * L1[ne]) <= tol * np.linalg.norm(L2[ne])


@pytest.mark.parametrize("limit", [1, 1000, 3000])
@pytest.mark.parametrize("P", [4, 16])
def test_tensorcore_m2l_wait_timeout_with_copies_in_flight(P, limit, tb, ctx):
    """Wait bounds around the time a copy takes, on lists of at most a tile or two per
    CTA: the copying warp may have left its loop before another role gives up, and
    its copies still have to land before the CTA ends.  Either the call reports the
    timeout or it succeeds, and the next call with the default bound is right."""
    x, y, z, q = tb.datasets.make("uniform_cube", 6000, 62)
    ctx.partition(x, y, z, q, ncrit=32)
    ctx.upward(P, tb.FP64)
    ctx.build_lists(0.5)
    ctx.m2l(tb.FP64)
    _, L64 = ctx.expansions()
    try:
        ctx.set_wait_limit(limit)
        for _ in range(3):
            try:
                ctx.m2l(tb.MIXED)
            except tb.TapasError as e:
                assert e.code == tb._lib.ERR_TIMEOUT
    finally:
        ctx.set_wait_limit(0)
    ctx.m2l(tb.MIXED)
    _, Lmx = ctx.expansions()
    ne = (ctx.cells()["nb"] > 0) & (np.linalg.norm(L64, axis=1) > 0)
    rel = np.linalg.norm(Lmx[ne] - L64[ne], axis=1) / np.linalg.norm(L64[ne], axis=1)
    assert rel.max() < 2e-5


def _clustered(tb, n, clusters, seed=92):
    """A cube with clusters far smaller than a cell of level 13, some bodies coincident."""
    x, y, z, q = [a.copy() for a in tb.datasets.make("uniform_cube", n, seed)]
    rng = np.random.default_rng(6)
    free = rng.permutation(n)
    for k, m in enumerate(clusters):
        idx, free = free[:m], free[m:]
        for a, c in ((x, 0.3), (y, -0.2), (z, 0.6)):
            a[idx] = c - 0.007 * k + 3e-6 * rng.random(m)
        for a in (x, y, z):
            a[idx[m // 2:m // 2 + 5]] = a[idx[0]]
    return x, y, z, q


@pytest.mark.parametrize("n,clusters,ncrit", [
    (2000, [33], 4), (4096, [33, 34, 1000], 4), (9000, [40] * 100, 16), (9000, [4096], 16),
    (9000, [4097, 33], 64), (40000, [40, 17000, 33, 9000], 64), (5000, [5000], 8),
    (70000, [35] * 300 + [30] * 300, 16)])
def test_tree_long_runs_of_close_bodies(n, clusters, ncrit, tb, ctx, oracle_mod):
    """Clusters whose bodies agree in all 40 key bits sorted first: longer than the
    insertion takes, one or many, few bodies or all, on both sides of the one-block
    sort's limit, against the oracle's tree, bit for bit."""
    _check_tree(tb, ctx, oracle_mod, *_clustered(tb, n, clusters), ncrit)


@pytest.mark.parametrize("n", [3000, 50000])
def test_long_runs_do_not_sort_everything_again(n, tb, ctx):
    """A few close bodies cost a sort of themselves (six launches more), not one of all
    bodies on all bits (24 passes' launches)."""
    launches = []
    for clusters in ([30], [33]):
        b = _clustered(tb, n, clusters)
        ctx.partition(*b, ncrit=64)
        ctx.kernel_launches(True)
        ctx.partition(*b, ncrit=64)
        launches.append(ctx.kernel_launches(True))
    assert launches[1] - launches[0] == 6


def _pair_codes(keys, order, t, s):
    """Sorted codes of (target, source) pairs, cells numbered by key (order: argsort)."""
    rank = np.empty(len(keys), np.int64)
    rank[order] = np.arange(len(keys))
    return np.sort(rank[t] * len(keys) + rank[s])


@pytest.mark.parametrize("mutual", [0, 1])
@pytest.mark.parametrize("n,ncrit,theta,over", [
    (3000, 16, 0.1, "frontier and P2P"), (40000, 16, 0.25, "frontier and M2L"),
    (3000, 16, 0.4, "none")])
def test_traversal_outgrows_its_first_buffers(n, ncrit, theta, over, mutual, tb, oracle_mod):
    """Lists and frontiers longer than a fresh context's buffers end the traversal's
    launch; it goes on from that step in larger ones.  The lists are the oracle's, from
    a context whose first traversal this is and from one that has grown from a
    smaller set's."""
    x, y, z, q = tb.datasets.make("uniform_cube", n, 21)
    o = oracle_mod.Oracle(x, y, z, q, P=2, ncrit=ncrit, theta=theta, mutual=mutual)
    okeys = o.cells()["key"]
    oo = np.argsort(okeys, kind="stable")
    expected = []
    for t, s in (o.m2l_list(), o.p2p_list()):
        if mutual:  # the unordered pairs, both ways
            other = t != s
            t, s = np.concatenate([t, s[other]]), np.concatenate([s, t[other]])
        expected.append(_pair_codes(okeys, oo, t, s))
    for small_first in (False, True):
        with tb.Context(0) as c:
            c.set_reference_lists(True)
            if small_first:
                c.partition(*tb.datasets.make("uniform_cube", 200, 22), ncrit=16)
                c.build_lists(0.5, mutual)
            c.partition(x, y, z, q, ncrit=ncrit)
            launches = []
            for _ in range(2):
                c.kernel_launches(True)
                info = c.build_lists(theta, mutual)
                launches.append(c.kernel_launches(True))
                keys = c.cells()["key"]
                go = np.argsort(keys, kind="stable")
                for got, want in zip(c.lists(), expected):
                    assert np.array_equal(_pair_codes(keys, go, *got), want)
            assert (launches[0] > launches[1]) == (over != "none")
            first = 1.125 * (128 * len(keys) + 4096) + 1024
            assert (info["n_m2l"] / (1 + mutual) > first) == ("M2L" in over)


def test_first_traversal_of_the_default_cube_runs_through(tb):
    """100k bodies of a cube at the default setting fit a fresh context's buffers."""
    with tb.Context(0) as c:
        c.partition(*tb.datasets.make("uniform_cube", 100000, 3), ncrit=64)
        launches = []
        for _ in range(2):
            c.kernel_launches(True)
            c.build_lists(0.4)
            launches.append(c.kernel_launches(True))
        assert launches[0] == launches[1]


@contextlib.contextmanager
def _free_memory(mb):
    """The GPU's memory taken but for about `mb` MiB."""
    import torch
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    rest = torch.cuda.mem_get_info()[0] - (mb << 20)
    hog = torch.empty(rest, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hog
        torch.cuda.empty_cache()


def test_out_of_memory_is_reported_once(tb):
    """An allocation that fails is its own call's error, not also that of the next
    call's first launch."""
    b = tb.datasets.make("sphere_surface", 1000000, 9)
    with tb.Context(0) as c:
        c.partition(*b, ncrit=128)
        with _free_memory(24):
            with pytest.raises(tb.TapasError) as e:
                c.build_lists(0.4)
            assert e.value.code == tb._lib.ERR_NOMEM
        c.partition(*b, ncrit=128)
        assert c.build_lists(0.4)["n_p2p"] > 0


@pytest.mark.parametrize("mutual", [0, 1])
def test_lists_where_memory_is_short(mutual, tb):
    """Where the GPU's memory does not hold the traversal's first sizes (122 MB for
    this tree), it runs with what each step needs: the same lists."""
    b = tb.datasets.make("sphere_surface", 1000000, 9)
    with tb.Context(0) as c:
        c.partition(*b, ncrit=128)
        c.build_lists(0.4, mutual)
        want = c.lists()
    with tb.Context(0) as c:
        c.partition(*b, ncrit=128)
        with _free_memory(80):
            c.build_lists(0.4, mutual)
            got = c.lists()
        for g, w in zip(got, want):
            assert np.array_equal(g[0], w[0]) and np.array_equal(g[1], w[1])


@pytest.mark.parametrize("mb", [850, 600])
def test_fp64_m2l_where_memory_is_short(mb, tb):
    """Where the GPU's memory does not hold the product rows' 512 MiB, the M2L takes
    shorter ranges and leaves the near field its room: the same bits."""
    b = tb.datasets.make("uniform_cube", 60000, 12)

    def evaluate(c):
        c.partition(*b, ncrit=16)
        c.upward(14, tb.FP64)
        with _free_memory(mb) if short else contextlib.nullcontext():
            c.traverse(0.35, precision=tb.FP64)
            c.downward(tb.FP64)
            return c.results()

    got = []
    for short in (False, True):
        with tb.Context(0) as c:
            got.append(evaluate(c))
    assert np.array_equal(*got)


@pytest.mark.parametrize("lo,hi", [(-30, 30), (-511.5, -510.5), (-537, -511.6), (-545, -538),
                                   (509.0, 511.99), (512.01, 514)])
def test_reciprocal_distance_within_its_bound(lo, hi, tb, ctx):
    """charge_over_distance by itself: one unit charge at the origin, chargeless bodies at
    distances 2^lo .. 2^hi, so a body's potential is 1/r alone.  In the ordinary
    range, with r^2 on both sides of the smallest normal number and near the
    largest, subnormal, zero (adds nothing) and infinite (nothing either).  Against
    extended precision, from the rounded r^2: the refined 1/sqrt is off by its last
    rounding (1/2 ulp), half the rounding of r^2 y (at most 1/2 ulp) and the
    series' rest (0.003 ulp); rsqrt, which takes the rest, by 1 ulp.  The acceleration has
    three such factors and three roundings."""
    rng = np.random.default_rng(17)
    n = 4000
    d = 2.0 ** rng.uniform(lo, hi, n) * rng.choice([-1.0, 1.0], n)
    x, q = np.concatenate([[0.0], d]), np.zeros(n + 1)
    q[0] = 1.0
    zero = np.zeros(n + 1)
    ctx.partition(x, zero, zero, q, ncrit=64)
    r = ctx.direct(np.arange(1, n + 1))
    with np.errstate(all="ignore"):
        r2 = d * d
        exact = np.where(r2 == 0, 0, 1 / np.sqrt(r2.astype(np.longdouble)))
    bound = np.spacing(np.maximum(exact.astype(np.float64), 1e-300)).astype(np.longdouble)
    assert np.all(np.abs(r[:, 0].astype(np.longdouble) - exact) <= 1.01 * bound)
    if lo >= -30 and hi <= 30:  # beyond, 1/r^3 leaves the FP64 range
        acc = -d.astype(np.longdouble) * exact ** 3
        assert np.all(np.abs(r[:, 1] - acc) <= 4.6 * 2.0 ** -52 * np.abs(acc))
        assert np.all(r[:, 2:] == 0)


@pytest.mark.parametrize("P", [3, 6, 16])
def test_one_body_feels_nothing(P, tb, ctx):
    """A single body's root cell has no width, and the body lies beside it: no field in
    either form."""
    one = [np.array([v]) for v in (0.3, 0.2, 0.7, 1.5)]
    for precision in (tb.FP64, tb.MIXED):
        r = ctx.evaluate(*one, P=P, ncrit=64, theta=0.4, precision=precision)
        assert np.array_equal(r, np.zeros((1, 4))), precision


@pytest.mark.parametrize("P", [4, 11])
def test_mixed_bodies_on_a_leafs_axis(P, tb, ctx):
    """Bodies of a lattice lie on the vertical axes through their leaves' centres.  The
    field there is finite in the mixed form wherever it is in the FP64 form (below the
    centre; at it and above it the reference's own angles give NaN)."""
    rng = np.random.default_rng(11)
    x, y, z = (rng.integers(-8, 9, (3, 4000)) / 8.0)
    q = rng.uniform(-1, 1, 4000)
    x[:2], y[:2], z[:2] = [-1, 1], [-1, 1], [-1, 1]
    r64 = ctx.evaluate(x, y, z, q, P=P, ncrit=16, theta=0.5, precision=tb.FP64)
    rmx = ctx.evaluate(x, y, z, q, P=P, ncrit=16, theta=0.5, precision=tb.MIXED)
    cells, (order, _) = ctx.cells(), ctx.sorted_bodies()
    on_axis = 0
    for c in np.flatnonzero((cells["leaf"] != 0) & (cells["nb"] > 0)):
        b = order[cells["bbeg"][c]:cells["bbeg"][c] + cells["nb"][c]]
        cx, cy, cz = cells["center"][c]
        on_axis += np.sum((x[b] == cx) & (y[b] == cy) & (z[b] < cz))
    assert on_axis > 0
    fine = np.isfinite(r64)
    assert np.isfinite(rmx[fine]).all()
    rows = fine.all(axis=1)
    num = np.linalg.norm(rmx[rows] - r64[rows], axis=0)
    assert np.all(num <= 2e-6 * np.linalg.norm(r64[rows], axis=0))

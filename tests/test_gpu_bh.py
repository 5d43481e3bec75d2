"""GPU: the Barnes-Hut path against the reference sample and the oracle.

Bars: FP64 form bit-exact (same operations in the same order as the sample);
FP32 form within 1e-5 relative of the FP64 form; accuracy against direct sum
below the reference's own gate (force and potential error < 1e-2,
test.sh:180-228)."""
import pathlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BH_GOLDEN = sorted((pathlib.Path(__file__).parent / "golden").glob("bh_*.npz"))


@pytest.mark.parametrize("path", BH_GOLDEN, ids=[p.stem for p in BH_GOLDEN])
def test_bh_fp64_bit_exact_against_reference(path, tb, ctx):
    g = np.load(path)
    r = ctx.bh_evaluate(g["x"], g["y"], g["z"], g["m"], ncrit=int(g["ncrit"]),
                        theta=float(g["theta"]), eps2=float(g["eps2"]), precision=tb.FP64)
    np.testing.assert_array_equal(r, g["bh"])


@pytest.mark.parametrize("ncrit", [1, 8, 32])
def test_bh_fp64_matches_oracle(ncrit, tb, ctx, oracle_mod):
    x, y, z, m = tb.datasets.make("plummer", 20000, 81)
    r = ctx.bh_evaluate(x, y, z, m, ncrit=ncrit, theta=0.5, eps2=1e-6, precision=tb.FP64)
    ref, cnt = oracle_mod.barnes_hut(x, y, z, m, ncrit=ncrit, theta=0.5, eps2=1e-6)
    np.testing.assert_array_equal(r, ref)
    na, nd = ctx.bh_counts()
    assert (na, nd) == (int(cnt[0]), int(cnt[1]))


def _bh_direct(x, y, z, m, tg, eps2):
    out = np.zeros((len(tg), 4))
    for k, i in enumerate(tg):
        dx, dy, dz = x - x[i], y - y[i], z - z[i]
        r2 = dx * dx + dy * dy + dz * dz + eps2
        ir = 1.0 / np.sqrt(r2)
        ir3 = ir ** 3
        out[k] = [np.sum(dx * ir3 * m), np.sum(dy * ir3 * m), np.sum(dz * ir3 * m),
                  np.sum(ir * m)]
    return out


def test_bh_fp32_and_accuracy(tb, ctx):
    x, y, z, m = tb.datasets.make("plummer", 50000, 82)
    r64 = ctx.bh_evaluate(x, y, z, m, ncrit=32, theta=0.5, eps2=1e-6, precision=tb.FP64)
    r32 = ctx.bh_evaluate(x, y, z, m, ncrit=32, theta=0.5, eps2=1e-6, precision=tb.MIXED)
    num = np.linalg.norm(r32 - r64, axis=0)
    den = np.linalg.norm(r64, axis=0)
    assert np.all(num / den < 1e-5)
    tg = tb.datasets.sample_targets(len(x), 200, seed=3)
    d = _bh_direct(x, y, z, m, tg, 1e-6)
    ef = np.sqrt(np.sum((r64[tg, :3] - d[:, :3]) ** 2) / np.sum(d[:, :3] ** 2))
    ep = np.sqrt(np.sum((r64[tg, 3] - d[:, 3]) ** 2) / np.sum(d[:, 3] ** 2))
    assert ef < 1e-2 and ep < 1e-2


@pytest.mark.parametrize("ncrit", [1, 3, 70])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 200, 3001])
def test_bh_walk_edges(n, ncrit, tb, ctx, oracle_mod):
    """Part-filled warps, a root that is a leaf, odd and even leaves, lists that
    end part-filled: FP64 bit-exact with the oracle, the FP32 walk with the
    same interaction counts and within its 1e-5 bar."""
    x, y, z, m = tb.datasets.make("plummer", n, 83)
    r = ctx.bh_evaluate(x, y, z, m, ncrit=ncrit, theta=0.6, eps2=1e-6, precision=tb.FP64)
    ref, cnt = oracle_mod.barnes_hut(x, y, z, m, ncrit=ncrit, theta=0.6, eps2=1e-6)
    np.testing.assert_array_equal(r, ref)
    assert ctx.bh_counts() == (int(cnt[0]), int(cnt[1]))
    r32 = ctx.bh_evaluate(x, y, z, m, ncrit=ncrit, theta=0.6, eps2=1e-6, precision=tb.MIXED)
    assert ctx.bh_counts() == (int(cnt[0]), int(cnt[1]))
    num, den = np.linalg.norm(r32 - r, axis=0), np.linalg.norm(r, axis=0)
    assert np.all(num <= 1e-5 * den)


@pytest.mark.parametrize("eps2", [1e-40, 0.0])
def test_bh_walk_softening_below_fp32(eps2, tb, ctx, oracle_mod):
    """A softening that is no normal FP32 number: every body meets itself at
    that distance, so the accelerations' and potentials' finiteness follows
    1/sqrt(eps2) in either precision (zero: not finite)."""
    x, y, z, m = tb.datasets.make("uniform_cube", 500, 84)
    r = ctx.bh_evaluate(x, y, z, m, ncrit=4, theta=0.5, eps2=eps2, precision=tb.FP64)
    ref, _ = oracle_mod.barnes_hut(x, y, z, m, ncrit=4, theta=0.5, eps2=eps2)
    np.testing.assert_array_equal(r, ref)
    r32 = ctx.bh_evaluate(x, y, z, m, ncrit=4, theta=0.5, eps2=eps2, precision=tb.MIXED)
    if eps2 > 0:  # 1/sqrt(1e-40) = 1e20 is an FP32 number, and dominates the potential
        ok = np.isfinite(r32[:, 3])
        assert ok.all()
        assert np.linalg.norm(r32[:, 3] - r[:, 3]) <= 1e-5 * np.linalg.norm(r[:, 3])
    else:
        assert not np.isfinite(r32[:, :3]).any()


def test_bh_massless_cells(tb, ctx, oracle_mod):
    """A far cluster without mass has no centre (0/0): the bodies that accept one
    of its cells get NaN, as in the sample; all others stay finite, in both
    precisions (an FP32 lane must not feel a cell that only its neighbours
    accept)."""
    x, y, z, m = [a.copy() for a in tb.datasets.make("uniform_cube", 3000, 85)]
    m[(x > 0.2) & (x < 0.5) & (y > 0)] = 0.0
    r = ctx.bh_evaluate(x, y, z, m, ncrit=4, theta=0.3, eps2=1e-6, precision=tb.FP64)
    ref, _ = oracle_mod.barnes_hut(x, y, z, m, ncrit=4, theta=0.3, eps2=1e-6)
    np.testing.assert_array_equal(r, ref)
    r32 = ctx.bh_evaluate(x, y, z, m, ncrit=4, theta=0.3, eps2=1e-6, precision=tb.MIXED)
    assert np.array_equal(np.isnan(r32), np.isnan(r))


@pytest.mark.parametrize("scale", [2.0 ** -3, 1.0, 2.0 ** 5])
@pytest.mark.parametrize("dx,eps2", [(1 - 2.0 ** -53, 2.0 ** -53), (1 - 2.0 ** -53, 1e-40),
                                     (2 - 2.0 ** -52, 2.0 ** -51), (1.0, 3 * 2.0 ** -52)])
def test_bh_fp64_distance_at_rounding_edge(dx, eps2, scale, tb, ctx, oracle_mod):
    """Squared distances next to a power of four, where the rounded square root has
    all mantissa bits set (or its exact value lies next to the middle of two numbers)
    and the reciprocal next to a middle: bit for bit the sample's."""
    x = np.array([0.0, dx * scale])
    zero, m = np.zeros(2), np.array([1.0, 3.0])
    args = dict(ncrit=1, theta=0.5, eps2=eps2 * scale * scale)
    r = ctx.bh_evaluate(x, zero, zero, m, precision=tb.FP64, **args)
    ref, _ = oracle_mod.barnes_hut(x, zero, zero, m, **args)
    np.testing.assert_array_equal(r, ref)


@pytest.mark.parametrize("ncrit", [1, 4])
def test_bh_fp32_unsoftened_potential_is_infinite(ncrit, tb, ctx):
    """eps2 = 0: every body meets itself at distance zero, so its potential is
    infinite (and no NaN) in either precision, whether its leaf is odd or even."""
    x, y, z, m = tb.datasets.make("uniform_cube", 500, 84)
    for precision in (tb.FP64, tb.MIXED):
        r = ctx.bh_evaluate(x, y, z, m, ncrit=ncrit, theta=0.5, eps2=0.0, precision=precision)
        assert np.all(r[:, 3] == np.inf), precision

"""Scheduled runs (small contractions sharing launches, T1 dressing in two passes) against the same operations one
by one: two iterations from T = 0 in both graph modes equal the eager ones.

Tolerance: every element is a sum of at most about 1e5 products of numbers below the block's largest, rounded in
another order; 1e-12 of the largest amplitude is that sum's FP64 rounding with room for two iterations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

T12 = ('T1A', 'T1B', 'T2A', 'T2B', 'T2C')


def _shapes(d, names):
    out = {}
    for b in names:
        n, nb = int(b[1]), 'ABCDE'.index(b[2])
        out[b] = (d.oa,) * (n - nb) + (d.ob,) * nb + (d.va,) * (n - nb) + (d.vb,) * nb
    return out


def _context(method, norb, occ_a, occ_b, froz, rhf=False, active=None):
    from ccq_b200 import integrals as I
    from ccq_b200 import lib, synth
    h, e2, _ = synth.generate(synth.SynthSpec(norb, 2 * occ_b, 2 * norb, 0.03, 77 + norb))
    fa, fb = I.fock(h, e2, occ_a, occ_b)
    v = I.spin_blocks(e2, froz)
    return lib.Context(froz, occ_a, occ_b, norb, method, fa, fb, *v, rhf=rhf, shift=0.5, active=active), \
        I.Dims(froz, occ_a, occ_b, norb)


def _modes(ctx, names, shapes, iterate=None):
    res = []
    for mode in (0, 1, 2):
        ctx.use_graph(mode)
        for b in names:
            ctx.set_block(b, np.zeros(shapes[b]))
        hist = [ctx.iterate(it)[:2] for it in (1, 2)]
        res.append((np.array(hist), {b: ctx.get_block(b, shapes[b]) for b in names}))
    return res


@pytest.mark.parametrize('method,norb,occ_a,occ_b,froz,rhf', [
    ('CCSD', 4, 2, 1, 0, False),      # items of one row
    ('CCSD', 9, 4, 3, 1, False),      # odd extents, frozen core
    ('CCSD', 31, 8, 8, 0, True),      # the largest block that is dressed by separate transforms
    # dressing in two passes: 4 and 6 occupied orbitals held per lane, odd extents, 8 (one tile exactly), 9
    # (a second tile, nearly empty), 12, 16 with different spins, 24
    ('CCSD', 32, 3, 3, 0, False),
    ('CCSD', 34, 6, 5, 0, False),
    ('CCSD', 33, 8, 8, 0, True),
    ('CCSD', 37, 9, 9, 0, False),
    ('CCSD', 36, 12, 11, 1, False),
    ('CCSD', 35, 15, 13, 0, False),
    ('CCSD', 40, 17, 17, 0, False),
    ('CCSD', 44, 25, 25, 0, False),   # beyond what the dressing passes hold
    ('CCSDT', 9, 3, 2, 0, False),
    ('CCSDT', 14, 4, 4, 0, True),
    ('CCSDTQ', 8, 4, 3, 0, False),
])
def test_scheduled_run_equals_operations(method, norb, occ_a, occ_b, froz, rhf):
    ctx, d = _context(method, norb, occ_a, occ_b, froz, rhf)
    names = T12 + (('T3A', 'T3B', 'T3C', 'T3D') if method != 'CCSD' else ()) + \
        (('T4A', 'T4B', 'T4C', 'T4D', 'T4E') if method == 'CCSDTQ' else ())
    shapes = _shapes(d, names)
    names = tuple(b for b in names if np.prod(shapes[b]))
    ref, *others = _modes(ctx, names, shapes)
    scale = max(np.abs(x).max() for x in ref[1].values())
    assert np.isfinite(scale) and scale > 0
    for hist, t in others:
        np.testing.assert_allclose(hist, ref[0], rtol=1e-11)
        for b in names:
            np.testing.assert_allclose(t[b], ref[1][b], atol=1e-12 * scale, rtol=0, err_msg=b)
    ctx.close()


def test_scheduled_active_space_and_pinned_kernel():
    """CCSDt (pieces of one contraction share an output) and force_tile (nothing merged) take the same steps."""
    ctx, d = _context('CCSDt', 12, 4, 4, 0, active=(2, 7))
    names = T12 + ('T3A', 'T3B', 'T3C', 'T3D')
    shapes = _shapes(d, names)
    ref, *others = _modes(ctx, names, shapes)
    ctx.force_tile(1)
    others += _modes(ctx, names, shapes)
    scale = max(np.abs(x).max() for x in ref[1].values())
    for hist, t in others:
        np.testing.assert_allclose(hist, ref[0], rtol=1e-11)
        for b in names:
            np.testing.assert_allclose(t[b], ref[1][b], atol=1e-12 * scale, rtol=0, err_msg=b)
    ctx.close()


@pytest.mark.parametrize('ds', [1, 2, 7, 12])
def test_diis_space(ds):
    """Two DIIS steps (the bordered system at its smallest, at odd sizes and at its largest) follow ccq's iteration:
    energies and residua of the dense oracle within the 1e-11 of the other trajectory tests."""
    from ccq_b200 import integrals as I
    from ccq_b200 import lib, synth
    from oracle.densecc import DenseCC
    h, e2, _ = synth.generate(synth.SynthSpec(6, 6, 12, 0.09, 5))
    fa, fb = I.fock(h, e2, 3, 3)
    v = I.spin_blocks(e2, 0)
    n = min(2 * (ds + 1), 15) + 1
    hist = DenseCC(fa, fb, *v, I.Dims(0, 3, 3, 6), 'CCSD').solve(diis_space=ds, max_iter=n, tol=0.0)[3]
    ctx = lib.Context(0, 3, 3, 6, 'CCSD', fa, fb, *v, diis_space=ds)
    ctx.use_graph(1)
    got = [ctx.iterate(it) for it in range(1, n + 1)]
    assert [g[2] for g in got] == [it % (ds + 1) == 0 for it in range(1, n + 1)]
    np.testing.assert_allclose([g[0] for g in got], [x[0] for x in hist], atol=1e-11, rtol=0)
    np.testing.assert_allclose([g[1] ** 2 for g in got], [x[2] ** 2 for x in hist], atol=1e-11, rtol=0)
    ctx.close()


def test_large_pageable_blocks_round_trip():
    """Blocks on both sides of the size that is copied by several threads, of odd lengths, and the whole vector."""
    ctx, d = _context('CCSDTQ', 12, 4, 3, 0)
    shapes = _shapes(d, ('T4A', 'T4B', 'T4C', 'T4D', 'T3B', 'T2B'))
    sizes = [8 * int(np.prod(s)) for s in shapes.values()]
    assert max(sizes) >= 2 * (4 << 20) and min(sizes) < 4 << 20
    rng = np.random.default_rng(3)
    put = {b: rng.normal(size=s) for b, s in shapes.items()}
    for b, x in put.items():
        ctx.set_block(b, x)
    for b, x in put.items():
        assert np.array_equal(ctx.get_block(b, shapes[b]), x), b
    t = rng.normal(size=ctx.t_size)
    ctx.set_t(t)
    assert np.array_equal(ctx.get_t(), t)
    ctx.close()


# Systems whose intermediates outgrow the accumulation buffers, so that contractions of 128 < K <= 256 which overwrite
# their output share launches: one item per tile (two K ranges would both store and lose half of the sum, an error
# of the order of the block itself).  Tolerance: per block, 1e-12 of its largest amplitude; sums of up to 1e5 terms
# rounded in another order differ by about sqrt(1e5) * 1.1e-16 = 4e-14 of the terms' root sum of squares, which leaves
# room for a cancellation of 30 and two iterations.
def _assert_same(ref, others):
    for hist, t in others:
        np.testing.assert_allclose(hist, ref[0], rtol=1e-11)
        for b in t:
            scale = np.abs(ref[1][b]).max()
            assert np.isfinite(scale) and scale > 0, b
            np.testing.assert_allclose(t[b], ref[1][b], atol=1e-12 * scale, rtol=0, err_msg=b)


@pytest.mark.parametrize('method,norb,occ_a,occ_b,froz,active', [
    ('CCSDt', 20, 5, 5, 0, (4, 7)),
    ('CCSDt', 20, 5, 5, 0, (3, 8)),
    ('CCSDT', 21, 6, 5, 0, None),
    ('CCSDT', 19, 7, 6, 0, None),
    ('CCSDT', 22, 7, 6, 1, None),
    ('CCSDTQ', 15, 5, 5, 0, None),
])
def test_overwriting_contractions(method, norb, occ_a, occ_b, froz, active):
    ctx, d = _context(method, norb, occ_a, occ_b, froz, active=active)
    names = T12 + ('T3A', 'T3B', 'T3C', 'T3D') + (('T4A', 'T4B', 'T4C', 'T4D', 'T4E') if method == 'CCSDTQ' else ())
    ref, *others = _modes(ctx, names, _shapes(d, names))
    _assert_same(ref, others)
    ctx.close()


@pytest.mark.parametrize('norb,occ_a,occ_b,rhf', [(9, 4, 3, False), (38, 7, 7, True), (33, 12, 11, False)])
def test_left_ranges(norb, occ_a, occ_b, rhf):
    """Left preparation, iterations and triples corrections of CR-CC(2,3) in the three modes; the corrections to 1e-11
    (products of two compared quantities, up to 3e7 of them summed)."""
    ctx, d = _context('CR-CC(2,3)', norb, occ_a, occ_b, 0, rhf)
    shapes = _shapes(d, T12)
    res = []
    for mode in (0, 1, 2):
        ctx.use_graph(mode)
        for b in T12:
            ctx.set_block(b, np.zeros(shapes[b]))
        e = [ctx.iterate(it)[0] for it in (1, 2)]
        if mode:   # the same T as the operations' own, so that what is compared is the left part
            for b in T12:
                ctx.set_block(b, t0[b])
        t0 = {b: ctx.get_block(b, shapes[b]) for b in T12}
        ctx.lambda_init(res[0][0][1] if mode else e[1])
        hist = e + [ctx.lambda_iterate(it)[0] for it in (1, 2)]
        parts = np.split(ctx.get_l(), np.cumsum([np.prod(shapes[b]) for b in T12])[:-1])
        lam = {b.replace('T', 'L'): x for b, x in zip(T12, parts)}
        res.append((np.array(hist), lam, ctx.crcc23()))
    _assert_same(res[0][:2], [r[:2] for r in res[1:]])
    assert np.all(np.abs(res[0][2]) > 0)
    for r in res[1:]:
        np.testing.assert_allclose(r[2], res[0][2], rtol=1e-11, atol=0)
    ctx.close()

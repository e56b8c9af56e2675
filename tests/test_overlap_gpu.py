"""The sorts of an overlap pass (csrc/overlap.cuh: in registers, or merging rows,
by tile and number of g-ordinates) on keys that their
words, which leave out the keys' low bits, cannot order by themselves, and on
keys already in order.  Integer results, so no tolerance: the sorted order of
every pass that is not the reference heapsort's is the stable order of the
mixed oracle, and bins and split positions are the oracle's in every pass."""
import numpy as np
import pytest

from helpers import JAC_TOL, RAD_TOL, assignment, jac_err, rad_err
from radtrancode_b200 import synth

pytestmark = pytest.mark.gpu


def _tables(kind, ng):
    kt = synth.make_ktables([synth.CH4, synth.C2H6], np_=6, nt=5, ng=ng, vmin=600.0, delv=0.4, nbin=4, seed=ng)
    a, b = kt.table(0), kt.table(1)
    g = np.arange(ng, dtype=np.float64) / (ng - 1)
    if kind == "flat":          # rows a few units in the last place apart, columns over many octaves
        a[...] = (a[..., :1] * (1.0 + 4e-7 * np.arange(ng))).astype(np.float32)
        b[...] = (b[..., :1] * 1e4 * 10.0 ** (9.0 * (g - 1.0))).astype(np.float32)
    elif kind == "wide":        # keys over about a hundred octaves
        a[...] = (a[..., :1] * 10.0 ** (28.0 * (g - 1.0))).astype(np.float32)
        b[...] = (b[..., :1] * 10.0 ** (29.0 * (g - 1.0))).astype(np.float32)
    elif kind == "apart":       # every row above the one before it: nothing to sort
        a[...] = (a[..., :1] * 10.0 ** (0.2 * np.arange(ng))).astype(np.float32)
        b[...] = (b[..., :1] * 1e-3 * (1.0 + g)).astype(np.float32)
    return kt


@pytest.mark.parametrize("kind", ["flat", "wide", "apart"])
@pytest.mark.parametrize("ng", [3, 11, 12, 16, 17, 20, 22])
@pytest.mark.parametrize("tile", [0, 8])     # 0: the wide tile, these calls having few wavenumbers
def test_order_of_close_keys(ctx, oracle, tile, kind, ng):
    kt, cia = _tables(kind, ng), synth.make_cia(ng)
    job = synth.make_job(kt, [synth.CH4, synth.C2H6], nlayer=13, seed=ng, nwave=4)
    job.amount[:, 3] = job.amount[:, 2]            # both gases' columns alike
    ctx.set_ktables(kt)
    ctx.set_cia(cia)
    ctx.set_debug(True)
    ctx.set_tile(tile)
    try:
        c, g, _ = ctx.cirsrtfg_wave(job)
        perm, split = ctx.debug_bins(job)
        st = ctx.stats()
    finally:
        ctx.set_debug(False)
        ctx.set_tile(0)
    _, (hperm, hsplit, _) = oracle.cirsrtfg_wave(kt, cia, job, oracle.ORC_MIXED, debug=True)
    assert st["sort_passes"] == int((hperm[..., 0] >= 0).sum()) > 0
    assert np.array_equal(split, hsplit)
    assert np.array_equal(assignment(perm, split, ng), assignment(hperm, hsplit, ng))
    oracle.lib().orc_set_sort_mode(1)
    try:
        _, (sperm, _, _) = oracle.cirsrtfg_wave(kt, cia, job, oracle.ORC_MIXED, debug=True)
    finally:
        oracle.lib().orc_set_sort_mode(0)
    other = (perm != sperm).any(axis=-1)           # passes in another than the stable order
    assert other.sum() <= st["exact_passes"]
    assert np.array_equal(perm[other], hperm[other])
    c64, g64, _ = oracle.cirsrtfg_wave(kt, cia, job, oracle.ORC_FP64)
    assert rad_err(c, c64) <= RAD_TOL
    assert jac_err(g, g64, job.nv) <= JAC_TOL


# quadrature weights (in 32nds) with ordinates broad enough for an element to cross two boundaries of the narrow bins
_BROAD = {4: [12, 4, 4, 12], 5: [12, 2, 4, 2, 12], 6: [12, 2, 2, 2, 2, 12], 8: [12, 1, 1, 2, 2, 1, 1, 12],
          9: [12, 1, 1, 1, 2, 1, 1, 1, 12], 10: [12] + [1] * 8 + [12], 20: [11] + [0.5] * 16 + [1, 1] + [11]}


def _case_of_gases(monkeypatch, ng, nabs, delg=None):
    """nabs absorbers of like strength, k nearly even in g, and the tables' weights."""
    gases = [(50 + k, 0) for k in range(nabs)]
    for gas in gases:
        monkeypatch.setitem(synth.VMR, gas, 1e-4)
    kt = synth.make_ktables(gases, np_=6, nt=5, ng=ng, nbin=8, seed=3)
    if delg is not None:
        kt.delg[:] = delg
        kt.g_ord[:] = np.cumsum(kt.delg) - kt.delg / 2
    rng = np.random.default_rng(3)
    for i in range(nabs):
        t = kt.table(i)
        first = 1.0 + 0.05 * rng.standard_normal(t[..., :1].shape)
        t[...] = 0.01 * first * np.cumsum(rng.uniform(0.6, 1.4, t.shape), axis=-1) / ng
    return kt, synth.make_cia(3), synth.make_job(kt, gases, nlayer=11, seed=3, nwave=6, vmr_perturb=0.1)


def _two_boundaries(perm, delg):
    """Passes of a capture in which one element reaches two bins' upper boundaries."""
    ng = len(delg)
    w = np.multiply.outer(delg, delg).ravel()           # REAL products
    g_ord = np.cumsum(delg.astype(np.float64))
    g_ord[-1] = max(g_ord[-1], 1.0)
    n = 0
    for p in perm.reshape(-1, ng * ng):
        if p[0] >= 0:
            sp = np.searchsorted(np.cumsum(w[p].astype(np.float64)), g_ord)
            n += bool(((sp[1:] == sp[:-1]) & (sp[1:] < ng * ng)).any())
    return n


@pytest.mark.parametrize("tile", [0, 8])
@pytest.mark.parametrize("ng,nabs", [(ng, n) for ng in (4, 5, 6, 8) for n in (2, 4, 7)] +
                         [(ng, n) for ng in (9, 10, 20) for n in (2, 4)])
def test_elements_across_two_boundaries(ctx, oracle, monkeypatch, ng, nabs, tile):
    """The sequential walk of rankg.f:118-152 with one to six gas columns
    before the last pass: every such pass is counted, and bins, radiance and
    Jacobian are the oracle's."""
    kt, cia, job = _case_of_gases(monkeypatch, ng, nabs, np.array(_BROAD[ng], np.float32) / 32)
    ctx.set_ktables(kt)
    ctx.set_cia(cia)
    ctx.set_debug(True)
    ctx.set_tile(tile)
    try:
        c, g, _ = ctx.cirsrtfg_wave(job)
        perm, split = ctx.debug_bins(job)
        st = ctx.stats()
    finally:
        ctx.set_debug(False)
        ctx.set_tile(0)
    _, (hperm, hsplit, _) = oracle.cirsrtfg_wave(kt, cia, job, oracle.ORC_MIXED, debug=True)
    assert st["irregular_passes"] == _two_boundaries(hperm, kt.delg) > 0
    assert np.array_equal(split, hsplit)
    assert np.array_equal(assignment(perm, split, ng), assignment(hperm, hsplit, ng))
    c64, g64, _ = oracle.cirsrtfg_wave(kt, cia, job, oracle.ORC_FP64)
    assert rad_err(c, c64) <= RAD_TOL
    assert jac_err(g, g64, job.nv) <= JAC_TOL


@pytest.mark.parametrize("tile", [0, 8])
@pytest.mark.parametrize("ng,nabs,nact,broad", [(5, 9, 8, False), (16, 10, 8, False), (20, 9, 8, False), (20, 9, 7, False),
                                                (4, 9, 8, True), (6, 9, 8, True)])
def test_eight_gas_columns(ctx, oracle, monkeypatch, ng, nabs, nact, broad, tile):
    """Seven and eight retrieved absorbers, no temperature, and further ones
    that are not retrieved: every column is rebinned in every pass, by the
    walk over bins and (broad) by the sequential one."""
    delg = np.array(_BROAD[ng], np.float32) / 32 if broad else None
    kt, cia, job = _case_of_gases(monkeypatch, ng, nabs, delg)
    job.xmap[:, 2 + nact:, :] = 0.0
    ctx.set_ktables(kt)
    ctx.set_cia(cia)
    ctx.set_tile(tile)
    try:
        c, g, _ = ctx.cirsrtfg_wave(job)
        st = ctx.stats()
    finally:
        ctx.set_tile(0)
    assert (st["irregular_passes"] > 0) == broad
    c64, g64, _ = oracle.cirsrtfg_wave(kt, cia, job, oracle.ORC_FP64)
    assert rad_err(c, c64) <= RAD_TOL
    assert jac_err(g, g64, job.nv) <= JAC_TOL

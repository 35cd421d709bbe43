"""Kernels at the sizes where their split of the work changes or leaves a remainder: cells that do not
fill a chunk or a tile, a mesh whose bins fill neither, packets per warp, lanes per cell."""
import numpy as np
import pytest

from conftest import synthetic_recpdf
from mocassin_xray_gb300 import abi, configs, Context, Setup

pytestmark = pytest.mark.gpu

COUNTS = ("crossings", "interactions", "absorptions", "scatterings", "escaped", "line_escapes", "emissions", "trapped")


def _temperatures(pattern, n, rng):
    i = np.arange(n)
    if pattern == "uniform":
        return np.full(n, 8000.0)
    if pattern == "drift":                       # chains that start apart are slow to meet
        return 5000.0 * np.exp(0.01 * np.abs((i + 300) % 600 - 300))
    if pattern == "creep":                       # within 10 % of each other for whole chunks
        return 9000.0 * (1.0 + 0.04 * np.sin(i / 90.0))
    return 8000.0 * np.where(rng.random(n) < 0.5, 1.0, 1.3)


@pytest.mark.parametrize("n", [3, 13, 33])
@pytest.mark.parametrize("pattern", ["uniform", "drift", "creep", "steps"])
def test_gaunt_cache_is_the_serial_chain(data_dir, oracle_lib, tmp_path, n, pattern):
    """The chunks' replay gives the cache's temperatures of the cells taken one after another: whole grids,
    then half of the cells left out by the skip rule."""
    s = Setup(configs.lognormal_gas(tmp_path / "ln", n=n, packets=1000), data_dir)
    rng = np.random.default_rng(n)
    te = s.get(abi.ARR_TE).copy()
    te[1:] = _temperatures(pattern, s.n_cells, rng)
    args = (s.info.nx, s.info.ny, s.info.nz, s.get(abi.ARR_ACTIVE))
    ctx = Context(0)
    ctx.load(s)
    ctx.put(abi.ARR_TE, te)
    ctx.opacity(1)
    compute = np.ones(s.n_cells + 1, np.uint8)
    compute[0] = 0
    ref, last = oracle_lib.gaunt_cache(*args, te, compute, -1.0)
    np.testing.assert_array_equal(ctx.get(abi.ARR_GAUNT_TE)[1:], ref[1:])
    keep = rng.random(s.n_cells + 1) < 0.5
    te2 = (te[::-1] if pattern != "drift" else te * 1.3).astype(np.float32)
    te2[0] = te[0]
    ctx.put(abi.ARR_TE, te2)
    ctx.put(abi.ARR_TEOLD, np.where(keep, te2, 2.0 * te2).astype(np.float32))
    ctx.put(abi.ARR_NEOLD, ctx.get(abi.ARR_NE))
    ctx.opacity(2)
    compute = (~keep).astype(np.uint8)
    compute[0] = 0
    ref, _ = oracle_lib.gaunt_cache(*args, te2, compute, last)
    on = compute != 0
    np.testing.assert_array_equal(ctx.get(abi.ARR_GAUNT_TE)[on], ref[on])
    ctx.close()


@pytest.mark.parametrize("name", ["h_small", "lognormal_small"])
def test_odd_mesh_matches_oracle(decks, data_dir, oracle_lib, name):
    """Opacity and emission on the reference's own mesh, whose bins fill neither a group of eight nor a tile of
    32, to the tolerances they meet on the configured meshes."""
    s = Setup(decks[name], data_dir, mesh_mode=abi.MESH_REFERENCE)
    assert s.info.nbins % 8 and s.info.nbins % 32
    rng = np.random.default_rng(5)
    te = s.get(abi.ARR_TE).copy()
    te[1:] = 6000.0 + 9000.0 * rng.random(s.n_cells)
    te = te.astype(np.float32)
    ne, ion = s.get(abi.ARR_NE), s.get(abi.ARR_IONDEN)
    ctx = Context(0)
    ctx.load(s)
    ctx.put(abi.ARR_TE, te)
    ctx.opacity(1)
    oo = oracle_lib.opacity(s, te=te, nthreads=4)
    np.testing.assert_allclose(ctx.get(abi.ARR_OPACITY)[:, 1:], oo[:, 1:], rtol=2e-5, atol=1e-35)
    ctx.emission(1)
    compute = np.ones(s.n_cells + 1, np.uint8)
    compute[0] = 0
    _, last = oracle_lib.gaunt_cache(s.info.nx, s.info.ny, s.info.nz, s.get(abi.ARR_ACTIVE), te, compute, -1.0)
    fl = oracle_lib.for_lines_emission(oracle_lib.BalanceTables(s), te, ne, ion.reshape(-1))
    ro, _ = oracle_lib.emission(s, last, te=te, ne=ne, ionden=ion.reshape(-1), for_lines=fl)
    np.testing.assert_allclose(ctx.get(abi.ARR_RECPDF)[:, 1:], ro[:, 1:], rtol=0, atol=3e-5)
    ctx.close()


@pytest.mark.parametrize("name", ["h_small", "lognormal_small", "xray_small"])
@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_FP32_GEOM])
def test_packets_per_warp_change_nothing(decks, data_dir, oracle_lib, name, precision):
    """One packet a lane (many blocks for the packets) and a warp's full slots (one block of 32 a SM, packets
    left to queue), with emissions at once and 32 at a time: the same events and, the sums being compensated,
    the same J bits; in FP64 the oracle's."""
    s = Setup(decks[name], data_dir)
    op = oracle_lib.opacity(s)
    rec = synthetic_recpdf(s.get(abi.ARR_NU), s.n_cells)
    tl = np.full(s.n_cells + 1, 0.3, np.float32)
    ctx = Context(0)
    ctx.load(s)
    for arr, v in ((abi.ARR_OPACITY, op), (abi.ARR_RECPDF, rec), (abi.ARR_TOTAL_LINES, tl)):
        ctx.put(arr, v)
    n, seed = 40000, 99
    st = ctx.transport(n, seed=seed, precision=precision)
    j = ctx.get(abi.ARR_JSTE)
    if precision == abi.PREC_FP64:
        jo, _, so = oracle_lib.transport(s, op, rec, tl, n=n, seed=seed, nthreads=4)
        np.testing.assert_array_equal(j, jo)
    for kw in (dict(block_size=32, grid_mult=1), dict(block_size=32, grid_mult=1, emit_batch=1),
               dict(block_size=96, grid_mult=1, emit_batch=32), dict(block_size=64, grid_mult=1, handoff_emissions=2)):
        s2 = ctx.transport(n, seed=seed, precision=precision, **kw)
        assert [getattr(s2, k) for k in COUNTS] == [getattr(st, k) for k in COUNTS], kw
        np.testing.assert_array_equal(ctx.get(abi.ARR_JSTE), j)
    ctx.close()


@pytest.mark.parametrize("deck", ["lognormal", "sphere"])
def test_lanes_per_cell_change_nothing(data_dir, tmp_path, deck):
    """The mixed balance gives a cell 32 lanes on small grids and eight, or four where there are few ions, from
    20 000 cells on; none of its sums depends on that: a nebula's cells are the same bits alone and in a batch."""
    p = (configs.lognormal_gas(tmp_path / "a", n=13, packets=20000, half_width=1.5e19) if deck == "lognormal"
         else configs.h_sphere(tmp_path / "a", n=19, packets=20000))
    s = Setup(p, data_dir)
    copies = 20000 // s.n_cells + 1
    sc, bc = Context(0), Context(0)
    sc.load(s)
    bc.load_batched([s] * copies)
    sc.opacity(1), bc.opacity(1)
    sc.emission(1), bc.emission(1)
    sc.transport(20000, seed=4)
    bc.transport_batched([20000] * copies, [4] * copies)
    for c in (sc, bc):
        c.normalize_j()
        c.balance(precision=abi.BAL_MIXED)
    for arr in (abi.ARR_TE, abi.ARR_NE, abi.ARR_N_ITER_T):
        one, all_ = sc.get(arr), bc.get(arr)
        for b in (0, copies - 1):
            np.testing.assert_array_equal(bc.nebula_cells(all_, b), one[1:])
    sc.close()
    bc.close()

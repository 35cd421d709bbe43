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


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_FP32_GEOM])
def test_packets_per_warp_change_nothing_in_a_batch(data_dir, tmp_path, precision):
    """The same over a ragged batch of octant and full grids: a warp's full slots with emissions at once and 32 at
    a time, one packet a lane, and each nebula alone give the same events and J bits."""
    decks = configs.nebula_batch(tmp_path, n=7, seed=5, octant_every=3, max_edge=13, packets_range=(2e3, 2e4))
    setups = [Setup(d, data_dir, mesh_mode=abi.MESH_LOG_EDGES) for d, _ in decks]
    packets = [pk for _, pk in decks]
    seeds = [70 + b for b in range(len(decks))]
    assert sum(packets) > 25000
    bc = Context(0)
    bc.load_batched(setups)
    bc.opacity(1)
    bc.emission(1)
    op, rec, tl = (bc.get(a) for a in (abi.ARR_OPACITY, abi.ARR_RECPDF, abi.ARR_TOTAL_LINES))
    st = bc.transport_batched(packets, seeds, precision=precision)        # one packet a lane: many blocks
    j = bc.get(abi.ARR_JSTE)
    for kw in (dict(emit_batch=1), dict(emit_batch=32), dict(emit_batch=7)):
        s2 = bc.transport_batched(packets, seeds, precision=precision, block_size=32, grid_mult=1, **kw)
        assert [getattr(s2, k) for k in COUNTS] == [getattr(st, k) for k in COUNTS], kw
        np.testing.assert_array_equal(bc.get(abi.ARR_JSTE), j)
        ms = bc.batch_transport_ms()
        assert np.all(ms > 0) and ms.max() <= s2.kernel_ms * 1.05 + 0.05
    for b, s in enumerate(setups):
        sc = Context(0)
        sc.load(s)
        for arr, v in ((abi.ARR_OPACITY, op), (abi.ARR_RECPDF, rec), (abi.ARR_TOTAL_LINES, tl)):
            one = np.zeros(v.shape[:-1] + (s.n_cells + 1,), np.float32)
            one[..., 1:] = bc.nebula_cells(v, b)
            sc.put(arr, one)
        sc.transport(packets[b], seed=seeds[b], precision=precision)
        np.testing.assert_array_equal(sc.get(abi.ARR_JSTE)[:, 1:], bc.nebula_cells(j, b))
        sc.close()
    bc.close()


def test_mesh_too_long_for_the_guide(data_dir, oracle_lib, tmp_path):
    """A mesh above 8192 bins, whose re-emissions are drawn by bisection of the whole row."""
    s = Setup(configs.h_sphere(tmp_path / "s", n=5, packets=1000, edge=6.0e18, nbins=9000), data_dir,
              mesh_mode=abi.MESH_LOG_EDGES)
    assert s.info.nbins > 8192
    op = oracle_lib.opacity(s, nthreads=4)
    rec = synthetic_recpdf(s.get(abi.ARR_NU), s.n_cells)
    tl = np.full(s.n_cells + 1, 0.2, np.float32)
    ctx = Context(0)
    ctx.load(s)
    for arr, v in ((abi.ARR_OPACITY, op), (abi.ARR_RECPDF, rec), (abi.ARR_TOTAL_LINES, tl)):
        ctx.put(arr, v)
    st = ctx.transport(20000, seed=3, precision=abi.PREC_FP64)
    jo, _, so = oracle_lib.transport(s, op, rec, tl, n=20000, seed=3, nthreads=4)
    assert st.emissions == so.emissions > 20000 and st.crossings == so.crossings
    np.testing.assert_array_equal(ctx.get(abi.ARR_JSTE), jo)
    ctx.close()


def test_more_grain_kinds_than_a_block_takes(data_dir, oracle_lib, tmp_path):
    """66 grain kinds (two species of 33 sizes), which the grain balance takes in two rounds of 64."""
    deck = configs.dust_shell(tmp_path / "d", n=9, packets=20000)
    a = np.logspace(np.log10(0.005), np.log10(0.25), 33)
    (deck.parent / "grainsizes.dat").write_text("33 sizes\n" + "".join(
        f"{k + 1} {x:.6e} {x ** -3.5:.6e}\n" for k, x in enumerate(a)))
    s = Setup(deck, data_dir)
    T = oracle_lib.DustTables(s)
    C1 = s.n_cells + 1
    td0 = s.get(abi.ARR_TDUST)
    assert td0.size == 3 * 34 * C1
    ctx = Context(0)
    ctx.load(s)
    ctx.opacity(1)
    op_o, sca_o = oracle_lib.dust_opacity(T, s.get(abi.ARR_NDUST), td0)
    np.testing.assert_allclose(ctx.get(abi.ARR_OPACITY)[:, 1:], op_o[:, 1:], rtol=1e-6)
    ctx.emission(1)
    np.testing.assert_allclose(ctx.get(abi.ARR_DUSTPDF)[:, 1:], oracle_lib.dust_pdf(T, td0)[:, 1:], rtol=0, atol=2e-6)
    ctx.transport(20000, seed=9, precision=abi.PREC_FP64)
    ctx.normalize_j()
    j = ctx.get(abi.ARR_JSTE)
    ctx.balance()
    td_o, _, black_o, _ = oracle_lib.dust_t(T, j, td0)
    np.testing.assert_array_equal(ctx.get(abi.ARR_LG_BLACK)[1:], black_o[1:])
    np.testing.assert_allclose(ctx.get(abi.ARR_TDUST).reshape(-1, C1)[:, 1:], td_o.reshape(-1, C1)[:, 1:], rtol=1e-5)
    ctx.close()


def test_lanes_per_cell_change_nothing_in_xray_gas(data_dir, tmp_path):
    """The X-ray gas with seven stages (inner shells, Auger electrons, 51 pairs of element and ion) has eight lanes
    a cell in a batch of more than 20 000 cells and 32 alone."""
    p = configs.xray_gas(tmp_path / "x", n=11, packets=20000)
    p.write_text(p.read_text().replace("nstages 27", "nstages 7"))
    s = Setup(p, data_dir)
    copies = 20000 // s.n_cells + 1
    sc, bc = Context(0), Context(0)
    sc.load(s)
    bc.load_batched([s] * copies)
    for c in (sc, bc):
        c.opacity(1)
        c.emission(1, precision=abi.PHASE_MIXED)
    sc.transport(20000, seed=4)
    bc.transport_batched([20000] * copies, [4] * copies)
    for c in (sc, bc):
        c.normalize_j()
        c.balance(precision=abi.BAL_MIXED)
    for arr in (abi.ARR_TE, abi.ARR_NE, abi.ARR_IONDEN, abi.ARR_N_ITER_T):
        one, all_ = sc.get(arr), bc.get(arr)
        for b in (0, copies - 1):
            np.testing.assert_array_equal(bc.nebula_cells(all_, b), one[..., 1:])
    sc.close()
    bc.close()

"""What a user of the package has it do, as cases to be timed: whole Monte Carlo
iterations, the single phases of one (opacity, emission, transport, balance) at
the sizes and precisions the configurations, tests and benchmark use, batches
of nebulae and the adjoint.

A case is a dict of plain values.  `kind` says which entry point runs, `deck`
which synthetic model (mocassin_xray_gb300.configs), `n` its grid edge, `after`
how many iterations were run before the one that is measured.  The outputs are
the context's own device arrays (mcx_device_ptr) and what the calls return.
"""
from __future__ import annotations

import ctypes
import math
import shutil
import tempfile
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import numpy as np
import torch

from mocassin_xray_gb300 import DATA_DIR, Context, Setup, abi, configs

# outputGas forbidden lines (element, ion, lower, upper level) of the adjoint: [OIII] 5007, [NII] 6583, [SII] 6716
LINES = [(8, 3, 3, 4), (7, 2, 3, 4), (16, 2, 1, 3)]


def _case(name, kind, deck, n, packets=0, after=0, mesh="config", fp64=False, size=0):
    c = dict(kind=kind, deck=deck, n=n, packets=packets, after=after, mesh=mesh, fp64=fp64, size=size)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest model in use: a whole iteration of the 19^3 octant H sphere, 1e5 packets
        _case("iterate-sphere19", "iterate", "sphere", 19, packets=100_000, after=1),
        # opacity of every cell of the 41^3 nebula on the 600-bin mesh (each iteration's first phase)
        _case("opacity-lognormal41", "opacity", "lognormal", 41),
        # re-emission CDFs of the same grid, production precision
        _case("emission-lognormal41", "emission", "lognormal", 41),
        # the same phase as iterate_mc calls it (exact level populations), X-ray chemistry, the
        # reference's 1333-bin mesh, a small grid
        _case("emission-exact-xray15", "emission", "xray", 15, mesh="reference", fp64=True),
        # the transport of the benchmark's first iteration: bulk histories only
        _case("transport-lognormal41", "transport", "lognormal", 41, packets=10_000_000),
        # the transport of its later iterations: trapped histories
        _case("transport-lognormal41-late", "transport", "lognormal", 41, packets=10_000_000, after=5),
        # X-ray gas, later iteration: tens of thousands of trapped histories in a few cells' gas
        _case("transport-xray27-late", "transport", "xray", 27, packets=3_000_000, after=3),
        # ionisation and thermal balance of the 41^3 nebula, mixed precision
        _case("balance-lognormal41", "balance", "lognormal", 41, packets=1_000_000, after=1),
        # the same in FP64, as Context.balance() and iterate_mc run it by default, X-ray chemistry, odd size
        _case("balance-fp64-xray13", "balance", "xray", 13, packets=200_000, after=1, mesh="reference", fp64=True),
        # a whole iteration of a dust-only shell (grain opacity, emission, transport, temperatures)
        _case("iterate-dust61", "iterate", "dust", 61, packets=10_000_000),
        # an iteration of many small nebulae in one batched context, ragged sizes and packet counts
        _case("batch24", "batch", "batch", 33, packets=300_000, size=24),
        # derivatives of line luminosities with respect to every cell's density (the backward direction)
        _case("adjoint-lognormal11", "adjoint", "lognormal", 11, packets=200_000, after=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["iterate", "iterate", "opacity", "emission", "transport", "transport", "transport", "balance",
                       "balance", "lines", "batch", "adjoint"])
    odd = 2 * rng.randint(4, 18) + 1                      # 9 .. 37: a cell sits on the source of a full grid
    mesh = rng.choice(["config", "config", "reference"])
    if kind == "iterate":
        deck = rng.choice(["sphere", "lognormal", "xray", "slab", "dust"])
        n = rng.randint(7, 30) if deck in ("sphere", "slab") else min(odd, 31)
        return _case("", kind, deck, n, packets=_log(rng, 1e4, 2e6), after=0 if deck == "dust" else rng.randint(0, 2),
                     mesh=mesh)
    if kind in ("opacity", "emission"):
        deck = rng.choice(["lognormal", "xray"])
        fp64 = kind == "emission" and rng.random() < 0.4
        return _case("", kind, deck, min(odd, 13) if fp64 else odd, mesh=mesh, fp64=fp64)
    if kind == "transport":
        deck = rng.choice(["sphere", "lognormal", "lognormal", "xray", "slab", "dust"])
        fp64 = rng.random() < 0.2
        n = rng.randint(7, 30) if deck in ("sphere", "slab") else min(odd, 31)
        return _case("", kind, deck, n, packets=_log(rng, 1e4, 2e5 if fp64 else 4e6),
                     after=0 if fp64 or deck == "dust" else rng.randint(0, 4), mesh=mesh, fp64=fp64)
    if kind == "balance":
        deck = rng.choice(["sphere", "lognormal", "xray"])
        fp64 = rng.random() < 0.3
        n = rng.randint(7, 30) if deck == "sphere" else odd
        return _case("", kind, deck, min(n, 13) if fp64 else n, packets=_log(rng, 5e4, 1e6), after=rng.randint(0, 2),
                     mesh=mesh, fp64=fp64)
    if kind == "lines":
        return _case("", kind, rng.choice(["lognormal", "xray"]), min(odd, 21), mesh=mesh)
    if kind == "batch":
        return _case("", kind, "batch", min(odd, 33), packets=_log(rng, 3e4, 5e5), size=rng.randint(2, 24))
    return _case("", kind, "lognormal", min(odd, 13), packets=_log(rng, 5e4, 3e5), after=rng.randint(0, 1))


# ------------------------------------------------------------------ inputs

def _mesh_mode(case):
    return abi.MESH_REFERENCE if case["mesh"] == "reference" else abi.MESH_LOG_EDGES


def _setup(case, seed):
    d = Path(tempfile.mkdtemp(prefix="mcx_case_"))
    try:
        n, pk = case["n"], max(case["packets"], 1)
        if case["deck"] == "sphere":
            p = configs.h_sphere(d, n=n, packets=pk)
        elif case["deck"] == "lognormal":
            p = configs.lognormal_gas(d, n=n, packets=pk, seed=seed)
        elif case["deck"] == "xray":
            p = configs.xray_gas(d, n=n, packets=pk)
        elif case["deck"] == "slab":
            p = configs.plane_slab(d, ny=n, packets=pk)
        else:
            p = configs.dust_shell(d, n=n, packets=pk, seed=seed)
        return Setup(p, DATA_DIR, mesh_mode=_mesh_mode(case))
    finally:
        shutil.rmtree(d, ignore_errors=True)


def _gas(case, setup, seed):
    """A gas state as a run passes through: Te around 1e4 K, each element's ionic fractions spread over its
    stages, H mostly ionised with a neutral tail, the electrons that go with them."""
    rng = np.random.default_rng([seed, case["n"]])
    info = setup.info
    C1, S, E = info.n_cells + 1, info.nstages, max(info.n_elem_used, 1)
    xref, abun = setup.get(abi.SARR_ELEM_XREF), setup.get(abi.ARR_ELEM_ABUN)
    te = 10.0 ** rng.normal(4.0, 0.12, C1)
    ion = np.zeros((S, E, C1))
    peak = rng.uniform(1.0, 4.0, C1)                    # the stage that dominates in the cell
    for z in range(1, 31):
        e = xref[z - 1]
        if e <= 0:
            continue
        top = min(z + 1, S)
        st = np.arange(1, top + 1)[:, None]
        w = np.exp(-2.0 * (st - np.minimum(peak, top)[None, :]) ** 2) + 1e-9
        if z == 1:
            x0 = 10.0 ** rng.uniform(-5.0, -0.3, C1)
            w = np.stack([x0, 1.0 - x0])[:top]
        ion[:top, e - 1] = w / w.sum(axis=0)
    ion = ion.astype(np.float32)
    charge = sum((ion[1:min(z + 1, S), xref[z - 1] - 1].astype(np.float64)
                  * np.arange(1, min(z + 1, S))[:, None]).sum(axis=0) * float(abun[z - 1])
                 for z in range(1, 31) if xref[z - 1] > 0)
    ne = charge * setup.get(abi.ARR_HDEN)
    return te.astype(np.float32), np.maximum(ne, 1e-3).astype(np.float32), ion


class _State:
    """A loaded context, what the case does with it, and its device arrays."""

    def __init__(self, case, seed, ctx):
        self.case, self.seed, self.ctx = case, seed, ctx

    def array(self, arr_id):
        """The context's array as a tensor on its device memory (the tensor keeps the context)."""
        shape, dtype = self.ctx._shape(arr_id)
        ptr = ctypes.c_void_p()
        self.ctx._check(abi.lib().mcx_device_ptr(self.ctx._h, arr_id, ctypes.byref(ptr)))
        return torch.as_tensor(_OnDevice(self.ctx, ptr.value, shape, np.dtype(dtype)), device="cuda")


class _OnDevice:
    def __init__(self, ctx, ptr, shape, dtype):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": tuple(int(v) for v in shape), "typestr": dtype.str,
                                         "data": (ptr, False), "version": 3, "strides": None}


_PREC = {False: dict(transport_precision=abi.PREC_FP32_GEOM, balance_precision=abi.BAL_MIXED,
                     emission_precision=abi.PHASE_MIXED),
         True: dict(transport_precision=abi.PREC_FP64, balance_precision=abi.BAL_FP64,
                    emission_precision=abi.PHASE_EXACT)}


def prepare(case, seed):
    ctx = Context(0)
    s = _State(case, seed, ctx)
    kind = case["kind"]
    if kind == "batch":
        d = Path(tempfile.mkdtemp(prefix="mcx_case_"))
        try:
            # the nebulae go by the case (their grids set the outputs' shapes), the packets by the seed
            decks = configs.nebula_batch(d, n=case["size"], seed=case["size"], max_edge=case["n"],
                                         packets_range=(case["packets"] / 30.0, float(case["packets"])))
            ctx.load_batched([Setup(p, DATA_DIR, mesh_mode=_mesh_mode(case)) for p, _ in decks])
        finally:
            shutil.rmtree(d, ignore_errors=True)
        s.packets = [pk for _, pk in decks]
        s.seeds = [seed * 1000 + b for b in range(len(decks))]
        ctx.state_save(0)
        return s
    setup = _setup(case, seed)
    ctx.load(setup)
    for it in range(1, case["after"] + 1):
        ctx.iterate(case["packets"], n_iterate_mc=it, seed=seed, counter_base=it << 40)
    if kind in ("opacity", "emission", "lines"):
        te, ne, ion = _gas(case, setup, seed)
        ctx.put(abi.ARR_TE, te)
        ctx.put(abi.ARR_NE, ne)
        ctx.put(abi.ARR_IONDEN, ion)
        if kind == "emission":
            ctx.opacity(1)
    elif kind in ("transport", "balance", "adjoint"):
        it = case["after"] + 1
        ctx.opacity(it)
        ctx.emission(it, precision=abi.PHASE_MIXED)
        if kind != "transport":
            ctx.transport(case["packets"], seed=seed, counter_base=it << 40)
            ctx.normalize_j()
    ctx.state_save(0)
    ctx.sync()
    return s


# -------------------------------------------------------------------- runs

_COUNTS = ("crossings", "interactions", "absorptions", "scatterings", "escaped", "line_escapes", "trapped", "emissions")


def _counts(st):
    return {k: int(getattr(st, k)) for k in _COUNTS}


def _gas_out(s):
    return {k: s.array(a) for k, a in (("te", abi.ARR_TE), ("ne", abi.ARR_NE), ("ionden", abi.ARR_IONDEN),
                                       ("converged", abi.ARR_LG_CONVERGED), ("black", abi.ARR_LG_BLACK))}


def _iteration_out(s, st):
    out = dict(counts=_counts(st.transport), jste=s.array(abi.ARR_JSTE), escaped=s.array(abi.ARR_ESCAPED),
               opacity=s.array(abi.ARR_OPACITY))
    if s.case["deck"] == "dust":
        return dict(out, tdust=s.array(abi.ARR_TDUST), pdf=s.array(abi.ARR_DUSTPDF),
                    converged=s.array(abi.ARR_LG_CONVERGED), black=s.array(abi.ARR_LG_BLACK))
    return dict(out, **_gas_out(s), pdf=s.array(abi.ARR_RECPDF), total_lines=s.array(abi.ARR_TOTAL_LINES))


def run(s):
    c, ctx = s.case, s.ctx
    kind, fp64, it = c["kind"], c["fp64"], c["after"] + 1
    if kind == "iterate":
        ctx.state_restore(0)
        st = ctx.iterate(c["packets"], n_iterate_mc=it, seed=s.seed, counter_base=it << 40, **_PREC[fp64])
        return _iteration_out(s, st)
    if kind == "batch":
        ctx.state_restore(0)
        st = ctx.iterate_batched(s.packets, s.seeds, **_PREC[fp64])
        return _iteration_out(s, st)
    if kind == "opacity":
        ctx.opacity(1)
        return {"opacity": s.array(abi.ARR_OPACITY)}
    if kind == "emission":
        ctx.emission(1, precision=abi.PHASE_EXACT if fp64 else abi.PHASE_MIXED)
        return {"pdf": s.array(abi.ARR_RECPDF), "total_lines": s.array(abi.ARR_TOTAL_LINES)}
    if kind == "transport":
        st = ctx.transport(c["packets"], seed=s.seed, counter_base=it << 40,
                           precision=abi.PREC_FP64 if fp64 else abi.PREC_FP32_GEOM)
        return {"counts": _counts(st), "jste": s.array(abi.ARR_JSTE), "escaped": s.array(abi.ARR_ESCAPED)}
    if kind == "balance":
        ctx.state_restore(0)
        ctx.balance(precision=abi.BAL_FP64 if fp64 else abi.BAL_MIXED)
        return _gas_out(s)
    if kind == "lines":
        r = ctx.line_luminosities()
        return {k: r[k] for k in ("hbeta_vol", "hydro", "hei", "forb", "wav", "te_vol", "ion_vol")}
    ctx.state_restore(0)
    r = ctx.adjoint(LINES, precision=abi.BAL_MIXED)
    return {k: r[k] for k in ("L", "dL_dhden", "dte_dhden")}


# -------------------------------------------------------------------- work

_BINS = {"sphere": 400, "lognormal": 600, "xray": 800, "slab": 400, "dust": 215, "batch": 600}
_REFERENCE_BINS = {"sphere": 1132, "lognormal": 1311, "xray": 1333, "slab": 1132, "dust": 215, "batch": 1311}
_ELEM_STAGES = {"sphere": (1, 3), "lognormal": (7, 7), "xray": (10, 27), "slab": (2, 3), "dust": (0, 0), "batch": (2, 3)}
# forms of atom data (ions with level populations), photoionised shells and updates per packet of each deck
_IONS = {"sphere": 0, "lognormal": 22, "xray": 60, "slab": 0, "dust": 0, "batch": 0}
_SHELLS = {"sphere": 1, "lognormal": 60, "xray": 300, "slab": 3, "dust": 0, "batch": 3}


def work(case):
    """Bytes: each input array read once, each output written once.  Operations: of the closed forms per (cell, bin)
    and per (cell, ion), one ladder per T-iteration, ~60 per estimator update."""
    deck, kind = case["deck"], case["kind"]
    n = case["n"]
    cells = {"sphere": n ** 3 / 2.0, "slab": 25.0 * n, "dust": 0.5 * n ** 3,
             "batch": case["size"] * (0.6 * n) ** 3 / 2.0}.get(deck, float(n ** 3))
    bins = (_REFERENCE_BINS if case["mesh"] == "reference" else _BINS)[deck]
    E, S = _ELEM_STAGES[deck]
    grid = cells * bins
    gas = 4.0 * cells * (2 + E * S)
    packets = case["packets"] * (case["size"] / 3.0 if kind == "batch" else 1.0)
    op = (4.0 * grid + gas, grid * (20.0 + _SHELLS[deck]))
    em = (4.0 * grid + gas, grid * 60.0 + cells * _IONS[deck] * 5e3)
    tr = (24.0 * grid, packets * 14.0 * 60.0)
    ba = (8.0 * grid + 2 * gas, grid * _SHELLS[deck] * 2.0 + cells * 6.0 * (_IONS[deck] * 2e3 + E * S * 100.0))
    parts = {"opacity": [op], "emission": [em], "transport": [tr], "balance": [ba], "lines": [(gas, em[1])],
             "adjoint": [(8.0 * grid + 2 * gas, 15.0 * ba[1])]}.get(kind, [op, em, tr, ba])
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


# ------------------------------------------------- values in 64 bits (numpy)

# Hummer (1988, ApJ 327, 477) Chebyshev coefficients of the free-free Gaunt factor, [11][8]
_HUMMER = np.array([
    8.986940175e+00, -4.009515855e+00, 8.808871266e-01, 2.640245111e-02, -4.580645915e-02, -3.568055702e-03,
    2.827798067e-03, 3.365860195e-04, -8.006936989e-01, 9.466021705e-01, 9.043402532e-02, -9.608451450e-02,
    -1.885629865e-02, 1.050313890e-02, 2.800889961e-03, -1.078209202e-03, -3.781305103e-01, 1.102726332e-01,
    -1.543619180e-02, 8.310561114e-03, 2.179620525e-02, 4.259726289e-03, -4.181588794e-03, -1.770208330e-03,
    1.877213132e-02, -1.004885705e-01, -5.483366378e-02, -4.520154409e-03, 8.366530426e-03, 3.700273930e-03,
    6.889320423e-04, 9.460313195e-05, 7.300158392e-02, 3.576785497e-03, -4.545307025e-03, -1.017965604e-02,
    -9.530211924e-03, -3.450186162e-03, 1.040482914e-03, 1.407073544e-03, -1.744671550e-03, 2.864013856e-02,
    1.903394837e-02, 7.091074494e-03, -9.668371391e-04, -2.999107465e-03, -1.820642230e-03, -3.874082085e-04,
    -1.707268366e-02, -4.694254776e-03, 1.311691517e-03, 5.316703136e-03, 5.178193095e-03, 2.451228935e-03,
    -2.277321615e-05, -8.182359057e-04, 2.567331664e-04, -9.155339970e-03, -6.997479192e-03, -3.571518641e-03,
    -2.096101038e-04, 1.553822487e-03, 1.509584686e-03, 6.212627837e-04, 4.098322531e-03, 1.635218463e-03,
    -5.918883504e-04, -2.333091048e-03, -2.484138313e-03, -1.359996060e-03, -5.371426147e-05, 5.553549563e-04,
    3.837562402e-05, 2.938325230e-03, 2.393747064e-03, 1.328839809e-03, 9.135013312e-05, -7.137252303e-04,
    -7.656848158e-04, -3.504683798e-04, -8.491991820e-04, -3.615327726e-04, 3.148015257e-04, 8.909207650e-04,
    9.869737522e-04, 6.134671184e-04, 1.068883394e-04, -2.046080100e-04]).reshape(11, 8)


def _clenshaw(c, x):
    """0.5 (b0 - b2) with the first coefficient halved, as the fit is defined."""
    b1 = b2 = 0.0
    for k in range(len(c) - 1, 0, -1):
        b1, b2 = x * b1 - b2 + c[k], b1
    b0 = x * b1 - b2 + c[0]
    return b0 - b2


def _gaunt(z_log10sq, te, nu):
    """Gaunt factor at temperatures te [T] (z_log10sq: log10 of the charge) and frequencies nu [B]: [B, T]."""
    lt = np.clip(np.log10(te), 2.5, 8.0)
    x = 5.1983649 - lt
    txg = 0.66666667 * (2.0 * z_log10sq + x)
    gamma2 = 10.0 ** (1.5 * txg)
    con = 0.72727273 * x + 0.90909091
    c = np.stack([0.25 * _clenshaw(_HUMMER[:, j], txg) for j in range(8)])      # [8, T]
    txu = 0.72727273 * np.log10(nu)[:, None] + con[None, :]
    u = 10.0 ** ((txu - 0.90909091) / 0.72727273)
    mid = _clenshaw([c[j][None, :] for j in range(8)], txu)
    g2 = np.broadcast_to(gamma2[None, :], txu.shape)
    low = np.where(g2 < 0.3, 0.551329 * np.log(2.24593 / u), 0.551329 * np.log(0.944931 / u / np.sqrt(g2)))
    lg = np.log10(g2)
    a, b = np.sqrt(0.9549297 / u), np.sqrt(12.0 * g2 / u)
    high = np.where(lg < -3.0, a, np.where(lg < 0.0, b + (b - a) / 3.0 * lg, np.minimum(1.05, b)))
    out = np.where(txu > 2.0, high, 0.0)
    out = np.where(np.log10(u) < -4.0, low, out)
    return np.where(np.abs(txu) <= 2.0, mid, out)


def _gaunt_temperatures(te):
    """BoltGaunt's cache: re-tabulated when Te moved by more than 10 % since the last tabulation, cells in order."""
    out, last = np.zeros(len(te), np.float32), np.float32(-1.0)
    for k in range(1, len(te)):
        if abs(np.float32(1.0) - last / te[k]) > np.float32(0.10):
            last = te[k]
        out[k] = last
    return out


def _xs(xsec, at):
    ok = (at >= 1) & (at <= len(xsec))
    return np.where(ok, xsec[np.clip(at, 1, len(xsec)) - 1], 0.0)


def _by_cells(f, n_cells, parts=16):
    """f(lo, hi) on chunks of the cells, in threads (numpy releases the interpreter); the results side by side."""
    cut = np.linspace(0, n_cells, min(parts, n_cells) + 1).astype(int)
    with ThreadPoolExecutor(max_workers=len(cut) - 1) as ex:
        return np.concatenate(list(ex.map(f, cut[:-1], cut[1:])), axis=1)


def _exact_opacity(case, seed):
    setup = _setup(case, seed)
    te32, ne, ion = _gas(case, setup, seed)
    info = setup.info
    nb, S = info.nbins, info.nstages
    nu, xsec = setup.get(abi.ARR_NU).astype(np.float64), setup.get(abi.ARR_XSEC).astype(np.float64)
    xref, abun = setup.get(abi.SARR_ELEM_XREF), setup.get(abi.ARR_ELEM_ABUN).astype(np.float64)
    P = setup.get(abi.SARR_POINTERS)
    eP = setup.get(abi.SARR_ELEMENT_P).reshape(30, 30, 7, 3)
    nsh = setup.get(abi.SARR_N_SHELLS).reshape(30, 30)
    hden = setup.get(abi.ARR_HDEN).astype(np.float64)
    te, ne = te32.astype(np.float64), ne.astype(np.float64)
    # the cross section of every ion at every bin, its shells added up
    ions, ff_weight = [], []
    for z in range(1, 31):
        if xref[z - 1] > 0:
            for i in range(1, min(z, S) + 1):
                ions.append((z, i))
                ff_weight.append((1.0 if i == 2 else 0.0) if z == 2 else float((i - 1) ** 2) if z >= 3 else 0.0)
    K = np.zeros((nb, len(ions)))
    for q, (z, i) in enumerate(ions):
        shells = ([(P[1], nb, P[0])] if z == 1 else [(P[3], nb, P[2]) if i == 1 else (P[5], nb, P[4])] if z == 2
                  else [tuple(int(v) for v in eP[z - 1, i - 1, sh]) for sh in range(nsh[z - 1, i - 1])])
        for lo, hi, first in shells:
            j = np.arange(max(lo, 1), min(max(lo, min(hi, nb)), nb) + 1)
            K[j - 1, q] += _xs(xsec, j + first - lo)
    gte = _gaunt_temperatures(te32).astype(np.float64)
    gte[0] = 1e4
    xb = xsec[np.arange(nb) + P[6] - 1][:, None]
    kn = setup.get(abi.ARR_KN_SIGMA_T).astype(np.float64)[:, None] if info.lg_compton else 0.0

    def part(lo, hi):
        t, n = te[lo:hi], ne[lo:hi]
        den = np.stack([ion[i - 1, xref[z - 1] - 1, lo:hi].astype(np.float64) * abun[z - 1] * hden[lo:hi] for z, i in ions])
        ff = (np.array(ff_weight) @ den) * n / 1e20 / np.sqrt(t)
        boltz = np.exp(-np.minimum(1.578866e5 / t + nu[:, None], 700.0))
        g = _gaunt(0.0, gte[lo:hi], nu)
        cont = np.where(boltz < 0.995, xb * (1.0 - boltz) * g, xb * nu[:, None] * g * 1.578866e5 / t)
        return K @ den + cont * ff + kn * n

    out = _by_cells(part, len(te))
    out[:, 0] = 0.0                                     # the dump cell is not computed
    return {"opacity": out}


def _exact_emission(case, seed):
    """The re-emission distribution (continua, HeI and HeII recombination and Lyman lines); totalLines needs every
    ion's level populations and is left out."""
    setup = _setup(case, seed)
    te32, ne32, ion = _gas(case, setup, seed)
    info = setup.info
    nb, S = info.nbins, info.nstages
    f64 = lambda a: setup.get(a).astype(np.float64)  # noqa: E731
    nu, xsec, abun = f64(abi.ARR_NU), f64(abi.ARR_XSEC), f64(abi.ARR_ELEM_ABUN)
    xref, P, dims = setup.get(abi.SARR_ELEM_XREF), setup.get(abi.SARR_POINTERS), setup.get(abi.SARR_EM_DIMS)
    tk, edge, lg = f64(abi.SARR_EM_TK), setup.get(abi.SARR_EM_EDGE_P).reshape(3, 32), f64(abi.SARR_EM_LOG_GAMMA)
    lg = lg.reshape(3, dims[0], 32)
    gte = np.array([_gaunt_temperatures(te32)[-1]], np.float64)
    hk, hc, con, four_pi = 157893.94, 2.1799153e-11, 4.9874105e-6, 4 * 3.141592654

    def part(lo, hi):
        te = te32[1 + lo:1 + hi].astype(np.float64)
        ne = np.maximum(ne32[1 + lo:1 + hi].astype(np.float64), 1e-5)
        x = lambda z, st: (ion[st - 1, xref[z - 1] - 1, 1 + lo:1 + hi].astype(np.float64)  # noqa: E731
                           if xref[z - 1] > 0 and st <= S else 0.0)
        sq, t15 = np.sqrt(te), te * np.sqrt(te)
        i1 = np.arange(1, nb + 1)
        # gamma(T, nu) of HI, HeI, HeII between the series edges
        pos = np.clip(np.searchsorted(tk, te) - 1, 0, dims[0] - 2)
        w = np.clip(np.log10(te / tk[pos]) / np.log10(tk[pos + 1] / tk[pos]), 0.0, 1.0)
        g = np.zeros((3, nb, len(te)))
        for k in range(3):
            loc = lg[k, pos] + (lg[k, pos + 1] - lg[k, pos]) * w[:, None]            # [T, 32]
            for p in range(1, dims[1 + k] // 2 + 1):
                up, low = edge[k, 2 * p - 1], edge[k, 2 * p - 2]
                a = (loc[:, 2 * p - 1] - loc[:, 2 * p - 2]) / (nu[up - 1] - nu[low - 1])
                j = np.arange(low, up)
                g[k, j - 1] = 10.0 ** (loc[:, 2 * p - 1][None, :] + a[None, :] * (nu[j - 1] - nu[up - 1])[:, None])
        ex = np.exp(-nu[:, None] * hk / te[None, :]) / sq[None, :]
        ff1 = four_pi * 54.43 * _gaunt(0.0, gte, nu) * ex
        ff2 = four_pi * 54.43 * 4.0 * _gaunt(0.30103, gte, nu) * ex
        start = [P[1], max(P[1], edge[1, dims[2] - 1])]
        start.append(max(start[1], edge[2, dims[3] - 1]))
        for k, (first, ip, stat, ff) in enumerate(((P[0], P[1], 2.0, ff1), (P[2], P[3], 0.5, ff1), (P[4], P[5], 2.0, ff2))):
            sel = i1 >= start[k]
            v = nu[sel][:, None]
            xs = _xs(xsec, i1[sel] - ip + first)[:, None]
            g[k, sel] = four_pi * xs * stat * hc * con * 1e40 * v ** 3 / t15 * np.exp((nu[ip - 1] - v) * hk / te) + ff[sel]
        heavy = np.zeros((nb, len(te)))
        for elem, stage, ip, high, first, g0, g1 in setup.get(abi.SARR_EM_FB_HEAVY).reshape(-1, 7):
            j = np.arange(max(ip, 1), min(high - 1, nb) + 1)
            xs = (_xs(xsec, j + first - ip) * (g0 / g1))[:, None]
            heavy[j - 1] += (np.exp((nu[ip - 1] - nu[j - 1])[:, None] * hk / te) * xs
                             * (x(elem, stage + 1) * abun[elem - 1]))
        heavy *= four_pi * con * hc * 1e40 * nu[:, None] ** 3 / t15
        # two-photon continua
        q = np.interp(np.log10(te), np.log10([1e4, 2e4]), np.log10([5.31e-4, 4.71e-4]))
        f_h = 0.8368 * (te * 1e-4) ** -0.723 / (1.0 + ne * 10.0 ** q / 8.23)
        f_he2 = 10.0 ** np.interp(np.log10(te), np.log10([5e3, 1e4, 1.5e4, 3e4]), np.log10([6.161, 4.091, 3.189, 2.035]))

        def shape(y):
            y = np.minimum(y, 1.0)
            return np.where(y < 1.0, 202.0 * (y * (1 - y) * (1 - (4 * y * (1 - y)) ** 0.8)
                                              + 0.88 * (y * (1 - y)) ** 1.53 * (4 * y * (1 - y)) ** 0.8) * y, 0.0)

        t_h = 6.6262e-27 * shape(nu / 0.7496) / 8.2249 * 1e27
        t_he2 = 6.6262e-27 * 0.9994667 * shape(nu / 3.0) / 8.226 * 1e27
        h2p = f64(abi.SARR_EM_HEI_2PHOT).reshape(2, 41)
        t_he1, j = np.zeros(nb), 1
        for i in range(nb):
            y = nu[i] / 1.514
            j += int(y > h2p[0, j - 1])
            if j >= 41:
                break
            a = h2p[1, j - 1] + (h2p[1, j] - h2p[1, j - 1]) / (h2p[0, j] - h2p[0, j - 1]) * (y - h2p[0, j - 1])
            t_he1[i] = (a if a >= 9.2163086e-3 else 0.0) * 0.66262 * y / 51.3
        wid = 3.2898423e15 * f64(abi.ARR_WIDFLX) / 1e15
        cut = lambda a: np.where(a < 1e-15, 0.0, a)  # noqa: E731
        tot = (cut((g[0] + t_h[:, None] * f_h) * (abun[0] * x(1, 2) * ne) + heavy * ne)
               + cut((g[1] + t_he1[:, None] * (6.23 * (te / 1e4) ** -0.827)) * (abun[1] * x(2, 2) * ne))
               + cut((g[2] + t_he2[:, None] * f_he2) * (abun[1] * x(2, 3) * ne))) * wid[:, None]
        tot[dims[6] - 1] += 27.2 * (te * 1e-4) ** -0.678 * ne * abun[1] * x(2, 2) * 1.45673 * 2.1799153e-11 * 1e11
        ly = f64(abi.SARR_EM_HEII_LYMAN)
        lya = 10.0 ** (-0.792 * np.log10(te) + 6.01) * ne * x(2, 3) * abun[1]
        for k in range(4):
            if 1 <= dims[7 + k] <= nb:
                tot[dims[7 + k] - 1] += lya * (1.0 if k == 3 else ly[k])
        cdf = np.cumsum(tot, axis=0)
        return cdf / cdf[-1]

    out = np.zeros((nb, len(te32)))
    out[:, 1:] = _by_cells(part, len(te32) - 1)
    return {"pdf": out, "total_lines": None}


def exact(case, seed):
    if case["kind"] == "opacity":
        return _exact_opacity(case, seed)
    if case["kind"] == "emission":
        return _exact_emission(case, seed)
    # a transport's histories and a balance's branches in 64 bits are other histories and branches
    return None

"""Calls at the edges of what the entry points take: what the caller reads back whole, memory, launches that fail
on the host, several threads, the largest axes, densities that are not numbers."""
import ctypes
import subprocess
import sys
import textwrap
from pathlib import Path

import numpy as np
import pytest

from conftest import synthetic_recpdf
from mocassin_xray_gb300 import abi, configs, Context, Setup

pytestmark = pytest.mark.gpu


# Host calls of the CUDA runtime that fail on request: fake_occupancy for a block size, fake_malloc for a size,
# fake_capturing a wait for the device, as while another thread captures a stream; and fake_attribute: an attribute
# of a kernel is set again to the least value that it ever had.
FAKES = r"""
#include <cstddef>
#include <map>
static int lowest = 0, capturing = 0;
static std::map<const void*, int> least;
static int occupancyOf = 0;
static size_t mallocOf = 0;
extern "C" {
void fake_occupancy(int blockSize) { occupancyOf = blockSize; }
void fake_malloc(size_t bytes) { mallocOf = bytes; }
void fake_attribute(int on) { lowest = on; }
void fake_capturing(int on) { capturing = on; }
int __real_cudaDeviceSynchronize(void);
int __wrap_cudaDeviceSynchronize(void) { return capturing ? 900 : __real_cudaDeviceSynchronize(); }
int __real_cudaFuncSetAttribute(const void*, int, int);
int __wrap_cudaFuncSetAttribute(const void* f, int attr, int value) {
  const int e = __real_cudaFuncSetAttribute(f, attr, value);
  auto at = least.emplace(f, value).first;
  if (value < at->second) at->second = value;
  return e || !lowest ? e : __real_cudaFuncSetAttribute(f, attr, at->second);
}
int __real_cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int*, const void*, int, size_t, unsigned);
int __wrap_cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int threads, size_t smem,
                                                                  unsigned flags) {
  if (occupancyOf && threads == occupancyOf) return 2;   // cudaErrorMemoryAllocation
  return __real_cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(n, f, threads, smem, flags);
}
int __real_cudaMalloc(void**, size_t);
int __wrap_cudaMalloc(void** p, size_t bytes) {
  if (mallocOf && bytes == mallocOf) return 2;
  return __real_cudaMalloc(p, bytes);
}
}
"""


@pytest.fixture(scope="module")
def fake_runtime(tmp_path_factory):
    """Runs a script in a process whose libmcx is this tree's, linked once more with FAKES in front of the
    runtime; fake(name, value) arms one of them."""
    from mocassin_xray_gb300 import _build
    d = tmp_path_factory.mktemp("fake")
    (d / "fake.cpp").write_text(FAKES)
    subprocess.run(["g++", "-O1", "-fPIC", "-c", "fake.cpp", "-o", "fake.o"], cwd=d, check=True)
    objs = sorted(str(o) for o in _build.BUILD.glob("*.o"))
    wraps = [x for f in ("cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags", "cudaMalloc", "cudaFuncSetAttribute",
                       "cudaDeviceSynchronize")
             for x in ("-Xlinker", f"--wrap={f}")]
    subprocess.run([_build._nvcc(), *_build.GENCODE, "-shared", "-o", str(d / "libfake.so"), *objs, str(d / "fake.o"),
                    *wraps, "-lpthread"], check=True)

    def run(script, *args):
        head = textwrap.dedent(f"""
            import ctypes, sys
            from pathlib import Path
            import numpy as np
            sys.path[:0] = [{str(Path(__file__).parent)!r}, {str(Path(__file__).parents[1])!r}]
            from conftest import DATA_DIR, synthetic_recpdf
            from mocassin_xray_gb300 import abi, configs, Context, Setup
            abi.LIB_PATH = Path({str(d / "libfake.so")!r})
            def fake(name, value): getattr(abi.lib(), "fake_" + name)(ctypes.c_size_t(value))
            """)
        r = subprocess.run([sys.executable, "-c", head + textwrap.dedent(script), *map(str, args)],
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout

    return run


def test_transport_after_a_failed_launch_starts_clean(fake_runtime, decks):
    """A transport whose second kernel cannot be set up leaves nothing to the next one: the same J bits as
    without it (FP64 deposits, whose sums need the compensation)."""
    fake_runtime("""
        s = Setup(sys.argv[1], DATA_DIR)
        ctx = Context(0)
        ctx.load(s)
        rng = np.random.default_rng(1)
        ctx.put(abi.ARR_OPACITY, (1e-18 * (0.2 + rng.random((s.info.nbins, s.n_cells + 1)))).astype(np.float32))
        ctx.put(abi.ARR_RECPDF, synthetic_recpdf(s.get(abi.ARR_NU), s.n_cells))
        ctx.put(abi.ARR_TOTAL_LINES, np.full(s.n_cells + 1, 0.05, np.float32))
        def run(seed):
            ctx.transport(20000, seed=seed, precision=abi.PREC_FP64)
            return ctx.get(abi.ARR_JSTE)
        ref = run(7)
        assert ref.sum() > 0
        fake("occupancy", 32)
        try: run(8)
        except abi.McxError: pass
        else: raise SystemExit("the fake did not fail the launch")
        fake("occupancy", 0)
        np.testing.assert_array_equal(run(7), ref)
        """, decks["lognormal_small"])


def _mixed_iteration(ctx, s):
    ctx.load(s)
    ctx.opacity(1)
    ctx.emission(1, precision=abi.PHASE_MIXED)
    ctx.transport(20000, seed=3, precision=abi.PREC_FP64)
    j = ctx.get(abi.ARR_JSTE)
    ctx.normalize_j()
    ctx.balance(precision=abi.BAL_MIXED)
    return j


def test_mixed_balance_takes_no_mesh_sized_memory(data_dir, tmp_path):
    """A model that fits the device fits it in its balance too, and the transport after a mixed balance is
    the one without it."""
    import torch
    small = Setup(configs.h_sphere(tmp_path / "a", n=5, packets=1000), data_dir)
    s = Setup(configs.h_sphere(tmp_path / "s", n=51, packets=1000), data_dir, mesh_mode=abi.MESH_REFERENCE)
    mesh = 4 * s.info.nbins * (s.n_cells + 1)
    assert mesh > 200 << 20
    ctx = Context(0)
    _mixed_iteration(ctx, small)        # what the kernels need of the process is there
    ctx.load(s)
    free = torch.cuda.mem_get_info()[0]
    j = _mixed_iteration(ctx, s)
    assert free - torch.cuda.mem_get_info()[0] < mesh // 4
    ctx.transport(20000, seed=3, precision=abi.PREC_FP64)
    np.testing.assert_array_equal(ctx.get(abi.ARR_JSTE), j)
    ctx.close()


def test_gas_without_level_ions_takes_no_local_memory(fake_runtime, decks):
    """The mixed balance of a gas without multi-level ions launches no kernel that solves them, whose local
    memory is gigabytes of the device."""
    out = fake_runtime("""
        import torch
        s = Setup(sys.argv[1], DATA_DIR)
        ctx = Context(0)
        ctx.load(s)
        ctx.opacity(1)
        ctx.emission(1, precision=abi.PHASE_MIXED)
        ctx.transport(2000, seed=3)
        ctx.normalize_j()
        free = torch.cuda.mem_get_info()[0]
        st = ctx.balance(precision=abi.BAL_MIXED)
        assert st.cells_updated > 0
        print(free - torch.cuda.mem_get_info()[0])
        """, decks["h_small"])
    assert int(out) < 64 << 20


def test_transport_without_memory_for_the_guide(fake_runtime, decks):
    """Where the device has no room for the guide to the re-emission CDFs, the model loads all the same and
    the draws are the same."""
    fake_runtime("""
        s = Setup(sys.argv[1], DATA_DIR)
        rec = synthetic_recpdf(s.get(abi.ARR_NU), s.n_cells)
        rng = np.random.default_rng(1)
        op = (1e-18 * (0.2 + rng.random((s.info.nbins, s.n_cells + 1)))).astype(np.float32)
        def run(precision):
            ctx = Context(0)
            ctx.load(s)
            ctx.put(abi.ARR_OPACITY, op)
            ctx.put(abi.ARR_RECPDF, rec)
            ctx.put(abi.ARR_TOTAL_LINES, np.full(s.n_cells + 1, 0.05, np.float32))
            st = ctx.transport(20000, seed=7, precision=precision)
            return st.emissions, ctx.get(abi.ARR_JSTE)
        for precision in (abi.PREC_FP64, abi.PREC_FP32_GEOM):
            fake("malloc", 0)
            n, j = run(precision)
            fake("malloc", 2 * 129 * (s.n_cells + 1))
            m, k = run(precision)
            assert n == m > 20000
            np.testing.assert_array_equal(j, k)
        """, decks["lognormal_small"])


def _many_elements(root, n, stages, edge=5):
    """An X-ray gas of the first n elements with this many ionisation stages."""
    p = configs.xray_gas(root, n=edge, packets=1000, half_width=7e18)
    p.write_text(p.read_text().replace("nstages 27", f"nstages {stages}"))
    (p.parent / "abun_xray.in").write_text("".join(
        "1.\n" if z == 0 else "0.1\n" if z == 1 else f"{1e-4 if z < n else 0.}\n" for z in range(30)))
    return p


def test_models_of_different_size_in_two_threads(fake_runtime, decks, tmp_path):
    """A large model's kernels are launched although another thread's smaller model sets the limit of their
    shared memory in between (the fake does that after each setting)."""
    fake_runtime("""
        models = [Setup(p, DATA_DIR) for p in sys.argv[1:3]]
        ctxs = [Context(0) for _ in models]
        fake("attribute", 1)
        for c, s in zip(ctxs, models):
            c.load(s)
            c.opacity(1)
            c.emission(1, precision=abi.PHASE_MIXED)
            c.transport(500, seed=1, precision=abi.PREC_FP64)
        """, decks["h_small"], _many_elements(tmp_path / "m", 20, 20))


@pytest.mark.parametrize("handoff", [0, 2])
def test_fp64_transport_over_long_axes(data_dir, oracle_lib, tmp_path, handoff):
    """Axes whose FP64 walls do not fit a block's shared memory (26 000 cells along y), the histories kept or
    handed to the trapped-packet kernel: the oracle's events and J bits."""
    s = Setup(configs.plane_slab(tmp_path / "s", nx=3, ny=26000, nz=3, nbins=300, nu_max=25.0), data_dir,
              mesh_mode=abi.MESH_LOG_EDGES)
    C1, nb = s.n_cells + 1, s.info.nbins
    op = np.full((nb, C1), 3e-18, np.float32)
    nu = s.get(abi.ARR_NU).astype(np.float64)
    cdf = np.cumsum(np.where(nu >= 1.0, nu ** 3 * np.exp(-(nu - 1.0) / 0.3), 1e-3 * nu ** 0.5))
    cdf = (cdf / cdf[-1]).astype(np.float32)
    cdf[-1] = 1.0
    rec = np.repeat(cdf[:, None], C1, axis=1)
    tl = np.full(C1, 0.1, np.float32)
    ctx = Context(0)
    ctx.load(s)
    for arr, v in ((abi.ARR_OPACITY, op), (abi.ARR_RECPDF, rec), (abi.ARR_TOTAL_LINES, tl)):
        ctx.put(arr, v)
    st = ctx.transport(2000, seed=5, precision=abi.PREC_FP64, handoff_emissions=handoff or -1)
    jo, _, so = oracle_lib.transport(s, op, rec, tl, n=2000, seed=5, nthreads=8)
    assert st.crossings == so.crossings and st.interactions == so.interactions and st.escaped == so.escaped
    assert (st.handed_off > 0) == (handoff > 0)
    np.testing.assert_array_equal(ctx.get(abi.ARR_JSTE), jo)
    ctx.close()


@pytest.mark.parametrize("name", ["lognormal_small", "xray_small"])
def test_densities_that_are_not_finite(decks, data_dir, oracle_lib, name):
    """Ion fractions that are infinite or no numbers reach the bins of their open shells and thresholds, as in
    the oracle, and no other cell."""
    s = Setup(decks[name], data_dir)
    S, C1 = s.info.nstages, s.n_cells + 1
    xref = s.get(abi.SARR_ELEM_XREF)
    te, ne = s.get(abi.ARR_TE), s.get(abi.ARR_NE)
    ion = s.get(abi.ARR_IONDEN).reshape(S, -1, C1).copy()
    for cell, z, stage, v in ((5, 8, 3, np.inf), (6, 8, 2, np.inf), (9, 7, 2, np.nan),
                              (C1 - 1, 1, 2, np.inf), (40, 16, 4, np.inf), (41, 2, 2, -np.inf)):
        ion[stage - 1, xref[z - 1] - 1, cell] = v
    ctx = Context(0)
    ctx.load(s)
    ctx.put(abi.ARR_IONDEN, ion)
    ctx.opacity(1)
    with np.errstate(all="ignore"):
        oo = oracle_lib.opacity(s, ionden=ion.reshape(-1), nthreads=4)
    np.testing.assert_allclose(ctx.get(abi.ARR_OPACITY)[:, 1:], oo[:, 1:], rtol=2e-5, atol=1e-35)
    assert np.isinf(oo[:, 5]).any() and np.isnan(oo[:, 9]).any()
    compute = np.ones(C1, np.uint8)
    compute[0] = 0
    _, last = oracle_lib.gaunt_cache(s.info.nx, s.info.ny, s.info.nz, s.get(abi.ARR_ACTIVE), te, compute, -1.0)
    for precision in (abi.PHASE_EXACT, abi.PHASE_MIXED):
        ctx.emission(1, precision=precision)
        ro, _ = oracle_lib.emission(s, last, ionden=ion.reshape(-1))
        np.testing.assert_allclose(ctx.get(abi.ARR_RECPDF)[:, 1:], ro[:, 1:], rtol=0, atol=3e-5)
    ctx.close()


def test_mixed_balance_of_unreached_inner_shells(decks, data_dir):
    """A stage whose inner shells no photon reaches feeds nothing upwards, however large its fraction: infinite
    gives what 1e10 gives (both are clamped in the first step of the ladder)."""
    s = Setup(decks["lognormal_small"], data_dir)
    ctx = Context(0)
    ctx.load(s)
    ctx.opacity(1)
    ctx.emission(1, precision=abi.PHASE_MIXED)
    ctx.transport(100000, seed=3)
    ctx.normalize_j()
    j = ctx.get(abi.ARR_JSTE)
    dark = j[s.get(abi.ARR_NU) > 10.0].sum(axis=0) == 0.0
    ion = ctx.get(abi.ARR_IONDEN).reshape(s.info.nstages, -1, s.n_cells + 1).copy()
    ctx.state_save()
    got = []
    for v in (np.inf, 1e10):
        ctx.state_restore()
        ion[1, s.get(abi.SARR_ELEM_XREF)[7] - 1] = v          # O+
        ctx.put(abi.ARR_IONDEN, ion)
        ctx.balance(precision=abi.BAL_MIXED)
        got.append([ctx.get(a) for a in (abi.ARR_TE, abi.ARR_NE, abi.ARR_IONDEN)])
    lit = dark & (ctx.get(abi.ARR_LG_BLACK) == 0)
    lit[0] = False                                              # no cell
    assert lit.sum() > 500
    for a, b in zip(*got):
        np.testing.assert_array_equal(a[..., lit], b[..., lit])
    ctx.close()


def test_skipped_cells_keep_a_cdf_written_in_place(decks, data_dir):
    """A re-emission CDF that the caller writes through mcx_device_ptr is the one that cells draw from after an
    emission phase that skips them, as after mcx_put."""
    import torch
    s = Setup(decks["lognormal_small"], data_dir)
    shape = (s.info.nbins, s.n_cells + 1)
    rec = synthetic_recpdf(s.get(abi.ARR_NU), s.n_cells)
    rng = np.random.default_rng(1)
    op = (1e-18 * (0.2 + rng.random(shape))).astype(np.float32)
    ctx = Context(0)
    ctx.load(s)
    ctx.opacity(1)
    ctx.emission(1)
    for arr, old in ((abi.ARR_TE, abi.ARR_TEOLD), (abi.ARR_NE, abi.ARR_NEOLD)):
        ctx.put(old, ctx.get(arr))
    ctx.put(abi.ARR_OPACITY, op)
    ctx.put(abi.ARR_RECPDF, rec)
    ctx.transport(20000, seed=2)
    j = ctx.get(abi.ARR_JSTE)
    ctx.put(abi.ARR_RECPDF, np.ones(shape, np.float32))
    ptr = ctypes.c_void_p()
    ctx._check(abi.lib().mcx_device_ptr(ctx._h, abi.ARR_RECPDF, ctypes.byref(ptr)))
    view = type("View", (), {"__cuda_array_interface__": {"shape": shape, "typestr": "<f4", "data": (ptr.value, False),
                                                          "version": 3, "strides": None}})()
    torch.as_tensor(view, device="cuda").copy_(torch.from_numpy(rec))
    torch.cuda.synchronize()
    ctx.emission(2)
    ctx.transport(20000, seed=2)
    np.testing.assert_array_equal(ctx.get(abi.ARR_JSTE), j)
    ctx.close()


@pytest.mark.parametrize("stages", [25, 31])
def test_balance_of_every_element(data_dir, oracle_lib, tmp_path, stages):
    """All 30 elements with many stages: the FP64 balance against the oracle, and the mixed one against it within
    its bounds (Te and Ne to 1e-4 on the cells whose T-iteration took the same path)."""
    s = Setup(_many_elements(tmp_path / "m", 30, stages), data_dir)
    ctx = Context(0)
    ctx.load(s)
    ctx.opacity(1)
    ctx.emission(1, precision=abi.PHASE_MIXED)
    ctx.transport(50000, seed=5, precision=abi.PREC_FP64)
    ctx.normalize_j()
    j = ctx.get(abi.ARR_JSTE)
    ctx.state_save()
    T = oracle_lib.BalanceTables(s)
    te_o, ne_o, ion_o, _, _, nit_o, _ = oracle_lib.balance(T, j, *(ctx.get(a) for a in (
        abi.ARR_TE, abi.ARR_NE, abi.ARR_IONDEN)), nthreads=8)
    st = ctx.balance(precision=abi.BAL_FP64)
    assert st.cells_updated > 60
    np.testing.assert_array_equal(ctx.get(abi.ARR_N_ITER_T)[1:], nit_o[1:])
    np.testing.assert_allclose(ctx.get(abi.ARR_TE)[1:], te_o[1:], rtol=1e-6)
    ion, ref = ctx.get(abi.ARR_IONDEN).reshape(-1, s.n_cells + 1)[:, 1:], ion_o.reshape(-1, s.n_cells + 1)[:, 1:]
    np.testing.assert_allclose(ion[ref > 1e-10], ref[ref > 1e-10], rtol=1e-6)
    ctx.state_restore()
    ctx.balance(precision=abi.BAL_MIXED)
    same = np.flatnonzero(ctx.get(abi.ARR_N_ITER_T)[1:] == nit_o[1:]) + 1
    assert same.size >= 0.95 * s.n_cells
    np.testing.assert_allclose(ctx.get(abi.ARR_TE)[same], te_o[same], rtol=1e-4)
    np.testing.assert_allclose(ctx.get(abi.ARR_NE)[same], ne_o[same], rtol=1e-4)
    ctx.close()


@pytest.mark.parametrize("batched", [0, 1])
def test_load_while_another_thread_captures(fake_runtime, decks, batched):
    """A model loads while another context's thread captures its balance, when a wait for the device is refused."""
    fake_runtime("""
        s = Setup(sys.argv[1], DATA_DIR)
        ctx = Context(0)
        fake("capturing", 1)
        ctx.load_batched([s, s]) if int(sys.argv[2]) else ctx.load(s)
        ctx.opacity(1)
        assert np.isfinite(ctx.get(abi.ARR_OPACITY)).all()
        """, decks["h_small"], batched)


class _Dirty:
    """Device allocations of these sizes filled with NaN, every second one given back (the others are held
    until the end, so that the driver keeps the memory in use)."""

    def __init__(self, sizes):
        self.cu = ctypes.CDLL("libcuda.so.1")
        self.held = []
        for n in sizes:
            p = ctypes.c_uint64()
            assert self.cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(n)) == 0
            assert self.cu.cuMemsetD8_v2(p, ctypes.c_ubyte(0xff), ctypes.c_size_t(n)) == 0
            self.held.append(p)
        assert self.cu.cuCtxSynchronize() == 0
        for p in self.held[::2]:
            assert self.cu.cuMemFree_v2(p) == 0

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        for p in self.held[1::2]:
            assert self.cu.cuMemFree_v2(p) == 0


def test_arrays_read_whole_start_at_zero(decks, data_dir, tmp_path):
    """The dump row of the grain CDF and the residuals of cells not evaluated are 0, whatever the device
    memory held before the load."""
    s = Setup(configs.dust_shell(tmp_path / "d", n=9, packets=100), data_dir)
    ctx = Context(0)
    with _Dirty([4 * s.info.nbins * (s.n_cells + 1)] * 64):
        ctx.load(s)
    ctx.opacity(1)
    ctx.emission(1)
    pdf = ctx.get(abi.ARR_DUSTPDF)
    assert np.all(pdf[:, 0] == 0.0) and np.all(pdf[-1, 1:] == 1.0)
    ctx.close()
    s = Setup(decks["h_small"], data_dir)
    ctx = Context(0)
    with _Dirty([8 * (s.n_cells + 1)] * 256):
        ctx.load(s)
    assert np.all(ctx.get(abi.ARR_BAL_RESID) == 0.0)
    ctx.close()

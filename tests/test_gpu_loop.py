"""GPU: the resident solver loop (one cooperative launch per solver phase)
against the launch-per-kernel loop (QPHIX_B200_LOOP=0) of the same solvers.

A fixed, small number of iterations is compared, so that the results differ
by the rounding of differently ordered sums only: after n iterations of a
well-conditioned system (m = 0.3, condition number about 100) they agree to a
few hundred units of the storage's rounding (FP64 1e-12, FP32 1e-4 of the
largest component; 16-bit storages round both alike and add 2^-15 per
vector store, 1e-3).  The lattices are the smallest, ragged ones, and ones on
either side of the loop's rules: groups of 4..32 sites, eight or four parts a
site, links read once per site (mirrored).
"""
import numpy as np
import pytest

from conftest import fields, rel_err, synthetic
from fixedpoint import naik_phased

pytestmark = pytest.mark.gpu

# sites per parity 128, 256, 768, 2304 (ragged), 20736 (four parts in FP32),
# 32768 (mirrored FP32 and FP64; four parts in FP64)
DIMS = [(4, 4, 4, 4), (4, 8, 4, 4), (8, 4, 4, 12), (12, 8, 4, 12), (12, 12, 12, 24), (16, 16, 16, 16)]
MODES = {"double": 1e-12, "F": 1e-4, "single": 1e-4, "r12": 1e-4, "half-links": 1e-4, "half": 1e-3}


def _solve(lib, mode, links, src, parity, n, masses):
    prec = "F" if mode == "F" else "D"
    lib.set_inner_precision({"F": "double", "r12": "single", "r13": "single"}.get(mode, mode))
    lib.set_link_compression(mode in ("r12", "r13"))
    try:
        L = lib.create_L(prec, links)
        b = lib.create_V(prec, src, parity)
        xs = [lib.create_V(prec, np.zeros_like(src), parity) for _ in masses]
        if len(masses) == 1:
            it, info, _ = lib.invert(prec, L, xs[0], b, masses[0], parity=parity, max_iter=n, nrestart=1, resid=1e-30)
        else:
            it, info, _ = lib.invert_multi(prec, L, xs, b, masses, parity=parity, max_iter=n, nrestart=1, resid=1e-30)
        assert info.status == 0, lib.last_error()
        out = [lib.extract_V(prec, x, parity) for x in xs]
        for h in xs + [b]:
            lib.destroy_V(prec, h)
        lib.destroy_L(prec, L)
        return it, out
    finally:
        lib.set_inner_precision("double")
        lib.set_link_compression(False)


def _both(lib, monkeypatch, *args):
    monkeypatch.setenv("QPHIX_B200_LOOP", "0")
    ref = _solve(lib, *args)
    monkeypatch.delenv("QPHIX_B200_LOOP")
    return _solve(lib, *args), ref


@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("mode", list(MODES))
def test_cg_iterations(gpu, monkeypatch, dims, mode):
    lib = gpu.use(dims)
    parity = "odd" if dims[3] == 12 else "even"
    src = synthetic.gaussian_source(dims, seed=5, parity=parity)
    (it, x), (it0, x0) = _both(lib, monkeypatch, mode, fields(dims), src, parity, 12, [0.3])
    assert it == it0
    assert rel_err(x[0], x0[0]) < MODES[mode]


@pytest.mark.parametrize("dims", [(4, 4, 4, 4), (12, 8, 4, 12), (12, 12, 12, 24)], ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("mode", ["double", "F", "r12"])
def test_multishift_iterations(gpu, monkeypatch, dims, mode):
    """kLoopMs (FP64, FP32) and kLoopMsDefer (mixed)."""
    lib = gpu.use(dims)
    src = synthetic.gaussian_source(dims, seed=6, parity="even")
    masses = [0.5, 0.3, 0.4]
    (it, x), (it0, x0) = _both(lib, monkeypatch, mode, fields(dims), src, "even", 10, masses)
    assert it == it0
    for a, b in zip(x, x0):
        assert rel_err(a, b) < MODES[mode]


@pytest.mark.parametrize("mode", ["double", "F", "single"])
def test_backward_links_that_are_not_shifted_forward_links(gpu, monkeypatch, mode):
    """One backward link changed: the loop must read the caller's backward
    links, not the forward ones of their sites.  (The operator is then not
    Hermitian; the iterations are compared, not a solution.)"""
    dims = (16, 16, 16, 16)
    lib = gpu.use(dims)
    src = synthetic.gaussian_source(dims, seed=7, parity="even")
    links = dict(fields(dims))
    changed = dict(links, fatback=links["fatback"].copy())
    changed["fatback"][72 * 1234:72 * 1234 + 18] *= 1.5
    (_, x), (_, x0) = _both(lib, monkeypatch, mode, changed, src, "even", 6, [0.3])
    assert rel_err(x[0], x0[0]) < MODES[mode]
    _, y = _solve(lib, mode, links, src, "even", 6, [0.3])
    assert rel_err(y[0], x0[0]) > 30 * MODES["single" if mode != "double" else "double"]


@pytest.mark.parametrize("mode,kernel", [("double", "k_solver_loop"), ("F", "k_solver_loop"), ("r12", "k_small_loop")])
def test_barrier_wait_that_runs_out(gpu, mode, kernel):
    """A poll limit of zero ends the first grid barrier: every block stores the
    failure word and returns, and the call reports it.  A multi-shift solve
    launches no other kernel with bounded waits before its loop (FP64 and FP32
    shifts run in k_solver_loop, the deferred ones of a small lattice in
    k_small_loop).  The next solve is the one without a failure, bit for
    bit."""
    dims = (8, 8, 8, 8)
    lib = gpu.use(dims)
    src = synthetic.gaussian_source(dims, seed=8, parity="even")
    args = (lib, mode, fields(dims), src, "even", 10, [0.5, 0.3, 0.4])
    want = _solve(*args)
    try:
        assert lib.set_wait_limit(0) == 0
        with pytest.raises(AssertionError, match="grid barrier of the solver loop timed out"):
            _solve(*args)
        with pytest.raises(AssertionError, match="timed out"):  # (a tuned Dslash may be the first to wait)
            _solve(lib, mode, fields(dims), src, "even", 10, [0.3])
    finally:
        lib.set_wait_limit(-1)
    got = _solve(*args)
    assert got[0] == want[0]
    for a, b in zip(got[1], want[1]):
        assert np.array_equal(a, b)


# 65536 sites per parity: 151 MB of 18-real, 126 MB of 12- and 13-real and
# 75 MB of 16-bit links, all read once per site where they are mirrored
LARGE = (16, 16, 16, 32)
_large = {}


def _large_links(mode):
    if not _large:
        _large["links"] = synthetic.asqtad_links(LARGE, seed=1001, device="cuda")
    if mode == "r13" and "r13" not in _large:
        _large["r13"] = naik_phased(LARGE, _large["links"])
    return _large["r13" if mode == "r13" else "links"]


RECON = {"single": 0, "r12": 1, "r13": 2, "half-links": 0, "half": 0}


@pytest.mark.parametrize("changed", [None, "fatback", "lngback"])
@pytest.mark.parametrize("mode", list(RECON))
def test_mirrored_storages(gpu, monkeypatch, mode, changed):
    """Every inner storage where its links are read in their own site's block:
    the sign bits (12-real) and ratios (13-real) come from there too, and the
    16-bit records are read at other offsets.  With one backward link changed
    (a Naik link by its phase, which keeps it 13-real but not 12-real) the
    caller's backward links must be read."""
    lib = gpu.use(LARGE)
    links = _large_links(mode)
    recon = RECON[mode]
    if changed:
        links = dict(links, **{changed: links[changed].copy()})
        z = links[changed][72 * 4321:72 * 4321 + 18].view(np.complex128)
        z *= 1.5 if changed == "fatback" else np.exp(1.0j)
        if changed == "lngback" and mode == "r12":
            recon = 2
    src = synthetic.gaussian_source(LARGE, seed=9, parity="odd")
    (it, x), (it0, x0) = _both(lib, monkeypatch, mode, links, src, "odd", 8, [0.3])
    assert lib.last_stats().links_compressed == recon
    assert it == it0
    tol = {"r13": 1e-4}.get(mode, MODES.get(mode))
    assert rel_err(x[0], x0[0]) < tol


@pytest.mark.parametrize("mode", ["single", "r12", "r13"])
def test_mirrored_multishift(gpu, monkeypatch, mode):
    """The deferred shifts' loop (kLoopMsDefer) on mirrored links."""
    lib = gpu.use(LARGE)
    src = synthetic.gaussian_source(LARGE, seed=10, parity="even")
    (it, x), (it0, x0) = _both(lib, monkeypatch, mode, _large_links(mode), src, "even", 8, [0.5, 0.3, 0.4])
    assert it == it0
    for a, b in zip(x, x0):
        assert rel_err(a, b) < 1e-4


@pytest.mark.parametrize("mode", ["double", "F", "single", "r12", "r13", "half-links", "half"])
@pytest.mark.parametrize("masses", [[0.3], [0.5, 0.3, 0.4]], ids=["cg", "multishift"])
def test_eight_parts_in_four_phases(gpu, monkeypatch, mode, masses):
    """12^4 (10368 sites per parity): too large for the three-phase loop, eight
    parts a site, links that are not read as mirrored."""
    dims = (12, 12, 12, 12)
    lib = gpu.use(dims)
    links = naik_phased(dims, fields(dims)) if mode == "r13" else fields(dims)
    src = synthetic.gaussian_source(dims, seed=11, parity="even")
    (it, x), (it0, x0) = _both(lib, monkeypatch, mode, links, src, "even", 8, masses)
    assert it == it0
    for a, b in zip(x, x0):
        assert rel_err(a, b) < {"r13": 1e-4}.get(mode, MODES.get(mode))


@pytest.mark.parametrize("mode", ["double", "F", "r12"])
@pytest.mark.parametrize("masses", [[0.3], [0.5, 0.3, 0.4]], ids=["cg", "multishift"])
def test_loop_launches_are_counted(gpu, monkeypatch, mode, masses):
    """The count says which route a solve took: the loop, or the kernels with
    the loop switched off, a forced Dslash variant or kernel timing."""
    dims = (8, 8, 8, 8)
    lib = gpu.use(dims)
    src = synthetic.gaussian_source(dims, seed=12, parity="even")
    args = (lib, mode, fields(dims), src, "even", 10, masses)
    _solve(*args)
    assert lib.last_loop_launches() >= 1
    monkeypatch.setenv("QPHIX_B200_LOOP", "0")
    _solve(*args)
    assert lib.last_loop_launches() == 0
    monkeypatch.delenv("QPHIX_B200_LOOP")
    try:
        lib.set_dslash_variant(1)
        _solve(*args)
        assert lib.last_loop_launches() == 0
        lib.set_dslash_variant(-1)
        lib.set_kernel_timing(True)
        _solve(*args)
        assert lib.last_loop_launches() == 0
    finally:
        lib.set_dslash_variant(-1)
        lib.set_kernel_timing(False)

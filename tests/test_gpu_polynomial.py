"""Long runs (64 time steps or more) evaluate functions of a Hermitian H from
Chebyshev vectors over the whole run (tbpm_poly_kernels.cuh) instead of step by
step.  Every case is compared with the time-stepping CPU oracle on the same
inputs: FP64 to the relative 1e-10 of the other parity tests, FP32 states to
their 3e-5; calls that must keep time stepping (a non-Hermitian matrix, long
rows, a series that is not unitary) are compared the same way.
"""

import math

import numpy as np
import pytest

import tbplas_b200 as tb
from tbplas_b200 import _native as nat
from tbplas_b200.fortran import f2py
from oracle import oracle

from conftest import bessel_series, rel_err, unit_states

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-10, "fp32": 3e-5}


@pytest.fixture(autouse=True)
def _backend():
    f2py.set_backend(precision="fp64", batch=16, device=0, state_kind="exp", term_kernel=0,
                     use_graphs=True, vector_width=0, threads_per_block=0, rows_per_tile=0)
    yield
    f2py.set_backend(precision="fp64", batch=16, term_kernel=0, vector_width=0)


@pytest.fixture(scope="module")
def flake():
    """A ragged open sample with vacancies in a field."""
    s = tb.make_graphene_sample(19, 23, disorder=1.0, vacancy_rate=0.02, pbc=False, rescale=9.0,
                                seed=3)
    s.set_magnetic_field(60.0)
    return s.build_ham_csr()


def _random_hermitian(n, degree, seed):
    """A sparse Hermitian matrix with rows of very different lengths, unsorted
    columns, and its largest row sum below 0.95."""
    rng = np.random.default_rng(seed)
    rows = [dict() for _ in range(n)]
    for r in range(n):
        for c in rng.integers(0, n, rng.integers(0, degree)):
            if c != r:
                v = complex(rng.standard_normal(), rng.standard_normal())
                rows[r][int(c)] = v
                rows[int(c)][r] = v.conjugate()
        rows[r][r] = complex(rng.standard_normal())
    top = max(sum(abs(v) for v in row.values()) for row in rows)
    ip = np.zeros(n + 1, dtype=np.int32)
    ix, hv = [], []
    for r, row in enumerate(rows):
        keys = list(row)
        rng.shuffle(keys)
        ip[r + 1] = ip[r] + len(keys)
        ix += keys
        hv += [row[k] * 0.95 / top for k in keys]
    return ip, np.array(ix, dtype=np.int32), np.array(hv, dtype=np.complex128)


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("kernel", [0, 1, 2])
@pytest.mark.parametrize("ns", [1, 3, 16])
def test_dos_long_run(flake, prec, kernel, ns):
    """One launch for all terms (0), the grid-stride kernel (1), the ring (2);
    with the norm check inside the run."""
    h = flake
    wf0 = unit_states(ns, h.shape[0], seed=ns)
    bes = bessel_series(math.pi)
    f2py.set_backend(precision=prec, term_kernel=kernel)
    got, per = f2py.tbpm_dos_states(bes, h.indptr, h.indices, h.data, wf0, 130, 128, 1e-9,
                                    per_state=True)
    ref = oracle.tbpm_dos(bes, h.indptr, h.indices, h.data, 130, wf0=wf0)
    assert rel_err(got, ref) < TOL[prec]
    assert np.allclose(per.mean(axis=0), got, rtol=0, atol=1e-14)


@pytest.mark.parametrize("n,degree", [(1, 1), (2, 2), (37, 3), (700, 9), (3001, 14)])
@pytest.mark.parametrize("width", [0, 1])
def test_dos_long_run_of_general_matrices(n, degree, width):
    """Rows with no entries up to tens of them, unsorted columns."""
    ip, ix, hv = _random_hermitian(n, degree, seed=n)
    wf0 = unit_states(4, n, seed=5)
    bes = bessel_series(math.pi)
    for kernel in (0, 1, 2):
        f2py.set_backend(vector_width=width, term_kernel=kernel)
        got = f2py.tbpm_dos_states(bes, ip, ix, hv, wf0, 64, 128, 1e-9)
        ref = oracle.tbpm_dos(bes, ip, ix, hv, 64, wf0=wf0)
        assert rel_err(got, ref) < 1e-10


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("nx,ns", [(101, 1), (128, 2), (128, 16), (256, 1), (300, 3), (580, 2)])
def test_dos_long_run_block_shapes(prec, nx, ns):
    """From the last size of the cluster kernel to several items per thread of
    the largest blocks of the one-launch kernel, device-generated states."""
    s = tb.make_graphene_sample(nx, nx, disorder=1.0, rescale=9.0, seed=11)
    h = s.build_ham_csr()
    bes = bessel_series(math.pi)
    f2py.set_backend(precision=prec)
    got = f2py.tbpm_dos(bes, h.indptr, h.indices, h.data, 7, 64, ns, "", 0, 128, 1e-9)
    ref = oracle.tbpm_dos(bes, h.indptr, h.indices, h.data, 64, seed=7, n_samples=ns)
    assert rel_err(got, ref) < TOL[prec]


def test_dos_other_time_steps(flake):
    """Half and twice the usual time step, a negative one, and a rescale factor
    far above the spectral radius."""
    h = flake
    wf0 = unit_states(2, h.shape[0], seed=1)
    for z, scale in ((math.pi / 2, 1.0), (2 * math.pi, 1.0), (-math.pi, 1.0), (math.pi, 0.02)):
        bes = [(-1) ** k * b for k, b in enumerate(bessel_series(-z))] if z < 0 \
            else bessel_series(z)
        got = f2py.tbpm_dos_states(bes, h.indptr, h.indices, h.data * scale, wf0, 96, 90, 1e-9)
        ref = oracle.tbpm_dos(bes, h.indptr, h.indices, h.data * scale, 96, wf0=wf0)
        assert rel_err(got, ref) < 1e-10


def test_calls_that_keep_time_stepping(flake):
    """A non-Hermitian matrix, a row of 80 entries, a series cut at 1e-6 (its
    step is not unitary to rounding)."""
    h = flake
    n = h.shape[0]
    wf0 = unit_states(2, n, seed=2)
    bes = bessel_series(math.pi)
    skew = h.data.copy()
    skew[11] *= 1 + 1e-9
    cut = bessel_series(math.pi, precision=1e-6)
    star = np.zeros((n, n), dtype=complex)
    star[5, 100:180] = 0.005j
    star[100:180, 5] = -0.005j
    import scipy.sparse as sp
    hs = sp.csr_matrix(h + sp.csr_matrix(star)) * 0.9
    for b, ip, ix, hv in ((bes, h.indptr, h.indices, skew), (bes, hs.indptr, hs.indices, hs.data),
                          (cut, h.indptr, h.indices, h.data)):
        got = f2py.tbpm_dos_states(b, ip, ix, hv, wf0, 70, 200, 1e-9)
        ref = oracle.tbpm_dos(b, ip, ix, hv, 70, wf0=wf0)
        assert rel_err(got, ref) < 1e-10


def test_norm_errors_of_long_runs(flake):
    """What check_norm refuses is refused: a rescale factor below the spectral
    radius, a series that loses norm, a NaN in a state."""
    h = flake
    n = h.shape[0]
    wf0 = unit_states(2, n, seed=4)
    bes = bessel_series(math.pi)
    with pytest.raises(nat.NormError):
        f2py.tbpm_dos_states(bes, h.indptr, h.indices, h.data * 4.5, wf0, 80, 64, 1e-9)
    with pytest.raises(nat.NormError):
        f2py.tbpm_dos_states(np.asarray(bes) * (1 - 1e-8), h.indptr, h.indices, h.data, wf0, 80,
                             64, 1e-9)
    wf0[1, 3] = np.nan
    with pytest.raises(nat.NanError):
        f2py.tbpm_dos_states(bes, h.indptr, h.indices, h.data, wf0, 80, 64, 1e-9)
    got = f2py.tbpm_dos_states(bes, h.indptr, h.indices, h.data, wf0[:1], 80, 64, 1e-9)
    assert rel_err(got, oracle.tbpm_dos(bes, h.indptr, h.indices, h.data, 80,
                                        wf0=wf0[:1])) < 1e-10


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("ns", [1, 3, 4, 16])
def test_packed_realisations_long_run(prec, ns):
    samples = [tb.make_graphene_sample(nx, ny, disorder=w, vacancy_rate=v, rescale=10.0, seed=i)
               for i, (nx, ny, w, v) in enumerate([(6, 5, 0.0, 0.0), (9, 7, 1.5, 0.02),
                                                   (70, 40, 3.0, 0.01)])]
    packed = tb.pack_samples(samples)
    bes = bessel_series(math.pi)
    f2py.set_backend(precision=prec)
    corr, per = f2py.tbpm_dos_segmented(bes, packed.indptr, packed.indices, packed.data,
                                        packed.offsets, ns, 1337, 72, 64, 1e-9, per_state=True)
    for k, s in enumerate(samples):
        h = s.build_ham_csr()
        for b in range(ns):
            ref = oracle.tbpm_dos(bes, h.indptr, h.indices, h.data, 72,
                                  seed=1337 * (k * ns + b + 1), n_samples=1)
            assert rel_err(per[k, b], ref) < TOL[prec]
        assert np.allclose(corr[k], per[k].mean(axis=0), rtol=0, atol=1e-14)


@pytest.fixture(scope="module")
def sample():
    s = tb.make_graphene_sample(9, 11, disorder=1.0, rescale=9.0, seed=21)
    s.set_magnetic_field(30.0)
    return s


@pytest.mark.parametrize("n_t,log", [(64, [0, 64]), (150, [0, 1, 2, 17, 90, 149]),
                                     (80, [79, 80]), (300, [7, 299]),
                                     (1100, [3, 1100])])
def test_psi_t_jumps(sample, n_t, log):
    """One expansion per logged interval, with and without the norm check."""
    h = sample.build_ham_csr()
    psi0 = unit_states(1, h.shape[0], seed=41)[0]
    bes = bessel_series(math.pi)
    got = f2py.tbpm_psi_t(bes, h.indptr, h.indices, h.data, psi0, np.array(log), n_t, 128, 1e-9)
    ref = oracle.tbpm_psi_t(bes, h.indptr, h.indices, h.data, psi0, np.array(log), n_t)
    assert rel_err(got, ref) < 1e-10
    psi0[3] = np.nan
    with pytest.raises(nat.NanError):
        f2py.tbpm_psi_t(bes, h.indptr, h.indices, h.data, psi0, np.array(log), n_t, 60, 1e-9)


def _energies(s, tnr, limits):
    e = np.array([0.5 * i * s.energy_range / tnr - s.energy_range / 2. for i in range(2 * tnr)])
    return e, np.where((e >= limits[0]) & (e <= limits[1]))[0]


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("fp32", 5e-5)])
@pytest.mark.parametrize("ns,n_en", [(1, 1), (3, 9), (4, 70), (2, 300)])
def test_eigenstates_long_run(sample, prec, tol, ns, n_en):
    """1 to 300 energies: one to ten groups of energy tiles, odd state counts."""
    h = sample.build_ham_csr()
    wf = unit_states(ns, h.shape[0], seed=6)
    t_step = 2 * math.pi / sample.energy_range
    energies = np.linspace(-2.0, 2.0, n_en) + 0.01
    bes = bessel_series(math.pi)
    f2py.set_backend(precision=prec)
    got = f2py.tbpm_eigenstates_states(bes, h.indptr, h.indices, h.data, wf, 66, t_step, energies,
                                       64, 1e-9)
    ref = oracle.tbpm_eigenstates(bes, h.indptr, h.indices, h.data, 66, t_step, energies, wf0=wf)
    assert rel_err(got, ref) < tol


@pytest.mark.parametrize("ns,tnr,batch", [(1, 64, 16), (3, 89, 2), (5, 70, 16)])
def test_dc_long_run(sample, ns, tnr, batch):
    """Filters for phase 1, several steps per expansion in phase 2 (remainders
    of 16 steps and of 8-step projections), several batches."""
    ip, ix, hv, dx, dy = sample.build_ham_dxy()
    wf0 = unit_states(ns, ip.size - 1, seed=31)
    energies, sel = _energies(sample, tnr, (-2.0, 2.0))
    bes = bessel_series(math.pi)
    t_step = 2 * math.pi / sample.energy_range
    f2py.set_backend(batch=batch)
    dos, dc = f2py.tbpm_dccond_states(bes, ip, ix, hv, sample.rescale, dx, dy, wf0, tnr, t_step,
                                      energies, sel, 60, 1e-9)
    rdos, rdc = oracle.tbpm_dccond(bes, ip, ix, hv, sample.rescale, dx, dy, tnr, t_step, energies,
                                   sel, wf0=wf0)
    assert rel_err(dos, rdos) < 1e-10
    assert rel_err(dc, rdc) < 1e-10


def test_dc_long_run_without_energies(sample):
    ip, ix, hv, dx, dy = sample.build_ham_dxy()
    wf0 = unit_states(2, ip.size - 1, seed=31)
    bes = bessel_series(math.pi)
    args = (bes, ip, ix, hv, sample.rescale, dx, dy)
    t_step = 2 * math.pi / sample.energy_range
    none = np.zeros(0, dtype=np.int32)
    dos, dc = f2py.tbpm_dccond_states(*args, wf0, 64, t_step, np.zeros(3), none, 60, 1e-9)
    rdos, _ = oracle.tbpm_dccond(*args, 64, t_step, np.zeros(3), none, wf0=wf0)
    assert rel_err(dos, rdos) < 1e-10 and not dc.any()
    wf0[0, 0] = np.inf
    with pytest.raises(nat.NanError):
        f2py.tbpm_dccond_states(*args, wf0, 64, t_step, np.zeros(3), none, 60, 1e-9)


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("fp32", 2e-5)])
@pytest.mark.parametrize("ns,tnr,chk", [(1, 64, 200), (3, 70, 64), (4, 97, 2)])
def test_ac_long_run(sample, prec, tol, ns, tnr, chk):
    ip, ix, hv, dx, dy = sample.build_ham_dxy()
    wf0 = unit_states(ns, ip.size - 1, seed=21)
    bes = bessel_series(math.pi / 2)
    beta = sample.rescale / (tb.KB * 3000.0)
    f2py.set_backend(precision=prec)
    got = f2py.tbpm_accond_states(bes, beta, 0.05, ip, ix, hv, sample.rescale, dx, dy, wf0, tnr,
                                  2**15, 1e-12, chk, 1e-9)
    ref = oracle.tbpm_accond(bes, beta, 0.05, ip, ix, hv, sample.rescale, dx, dy, tnr, wf0=wf0)
    assert np.all(got[:, 0] == 0)
    assert rel_err(got, ref) < tol


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("fp32", 2e-5)])
def test_dyn_pol_long_run(sample, prec, tol):
    h = sample.build_ham_csr()
    pos = sample.orb_pos
    q = [[1.3, 0.2, 0.0], [0.0, 2.0, 0.0], [0.5, 0.5, 0.0]]
    wf = unit_states(3, h.shape[0], seed=5)
    bes = bessel_series(math.pi / 2)
    beta = sample.rescale / (tb.KB * 3000.0)
    f2py.set_backend(precision=prec)
    got = f2py.tbpm_dyn_pol_states(bes, beta, 0.0, h.indptr, h.indices, h.data, pos[:, 0],
                                   pos[:, 1], pos[:, 2], q, wf, 75, 2**15, 1e-12, 64, 1e-9)
    ref = oracle.tbpm_dyn_pol(bes, beta, 0.0, h.indptr, h.indices, h.data, pos[:, 0], pos[:, 1],
                              pos[:, 2], q, 75, wf0=wf)
    assert rel_err(got, ref) < tol


def test_steps_per_expansion_follow_the_free_memory():
    """The same AC run with less and less free device memory (16, 8 and 4 steps per
    expansion with windows of 32, 16 and 8 vectors, then step by step): equal to rounding."""
    import torch
    s = tb.make_graphene_sample(192, 192, disorder=1.0, rescale=9.0, seed=2)
    ip, ix, hv, dx, dy = s.build_ham_dxy()
    n = ip.size - 1
    wf0 = unit_states(8, n, seed=3)
    bes = bessel_series(math.pi / 2)
    beta = s.rescale / (tb.KB * 6000.0)
    vb = n * 24 * 16
    args = (bes, beta, 0.0, ip, ix, hv, s.rescale, dx, dy, wf0, 64, 2**15, 1e-12, 128, 1e-9)
    ctx = nat.Context(0)  # holds no buffers yet: the process-wide context is left aside
    nat._contexts, kept = {0: ctx}, nat._contexts
    try:
        want = f2py.tbpm_accond_states(*args)
        ctx.close()
        for blocks in (44, 30, 24, 16, 8):
            nat._contexts[0] = ctx = nat.Context(0)
            f2py._ctx()
            torch.cuda.synchronize()
            free, _ = torch.cuda.mem_get_info(0)
            hold = torch.empty(free - (2 << 30) - int(blocks * vb) - (64 << 20),
                               dtype=torch.uint8, device="cuda")
            got = f2py.tbpm_accond_states(*args)
            del hold
            torch.cuda.empty_cache()
            ctx.close()
            assert rel_err(got, want) < 1e-12
    finally:
        nat._contexts = kept


@pytest.mark.parametrize("ns,n_lim", [(1, 8.5), (2, 8.5), (7, 3.0), (9, 1.0), (16, 2.0)])
def test_dc_projection_shapes(sample, ns, n_lim):
    """States and energies around the chunks of the projection kernel (8 states,
    32 energies per warp, warps left over for row splits), in one batch."""
    ip, ix, hv, dx, dy = sample.build_ham_dxy()
    wf0 = unit_states(ns, ip.size - 1, seed=31)
    energies, sel = _energies(sample, 64, (-n_lim, n_lim))
    bes = bessel_series(math.pi)
    t_step = 2 * math.pi / sample.energy_range
    args = (ip, ix, hv, sample.rescale, dx, dy)
    got = f2py.tbpm_dccond_states(bes, *args, wf0, 64, t_step, energies, sel, 60, 1e-9)
    ref = oracle.tbpm_dccond(bes, *args, 64, t_step, energies, sel, wf0=wf0)
    again = oracle.tbpm_dccond(bes, *args, 64, t_step, energies, sel,
                               wf0=wf0 * (1 + 1e-16 * np.random.default_rng(0).standard_normal(
                                   wf0.shape)))
    # wide windows reach energies with hardly any states (test_gpu_dc_shapes.py):
    # there the oracle's own sensitivity to rounding is the bar
    assert rel_err(got[0], ref[0]) < 1e-10
    assert rel_err(got[1], ref[1]) < max(1e-10, 8 * rel_err(again[1], ref[1]))


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("fp32", 3e-5)])
@pytest.mark.parametrize("n,degree", [(150, 2), (221, 9)])
def test_currents_of_general_matrices(prec, tol, n, degree):
    """AC and DC currents on rows of no entry, of fewer and of more entries than
    the current kernels load together."""
    ip, ix, hv = _random_hermitian(n, degree, seed=n)
    rng = np.random.default_rng(n)
    pos = rng.standard_normal((2, n))
    rows = np.repeat(np.arange(n), np.diff(ip))
    dx, dy = pos[:, ix] - pos[:, rows]
    wf0 = unit_states(3, n, seed=21)
    bes = bessel_series(math.pi / 2)
    f2py.set_backend(precision=prec)
    got = f2py.tbpm_accond_states(bes, 8.0, 0.05, ip, ix, hv, 1.0, dx, dy, wf0, 64, 2**12, 1e-12,
                                  128, 1e-9)
    ref = oracle.tbpm_accond(bes, 8.0, 0.05, ip, ix, hv, 1.0, dx, dy, 64, wf0=wf0, nr_fermi=2**12)
    assert rel_err(got, ref) < tol
    if prec == "fp32":  # a DC value divides by a projection, which may be small
        return
    bes = bessel_series(math.pi)
    energies, sel = np.linspace(-0.4, 0.4, 9), np.arange(9)
    got = f2py.tbpm_dccond_states(bes, ip, ix, hv, 1.0, dx, dy, wf0, 64, math.pi, energies, sel,
                                  128, 1e-9)
    args = (bes, ip, ix, hv, 1.0, dx, dy, 64, math.pi, energies, sel)
    ref = oracle.tbpm_dccond(*args, wf0=wf0)
    again = oracle.tbpm_dccond(*args, wf0=wf0 * (1 + 1e-16 * rng.standard_normal(wf0.shape)))
    # two hundred such perturbations: a run's own rounding is below 2e-14
    assert rel_err(got[0], ref[0]) < tol
    assert rel_err(got[1], ref[1]) < max(tol, 200 * rel_err(again[1], ref[1]))

"""Long runs at the edges of what their routes accept: packed samples that are not
uncoupled, matrices that are Hermitian to rounding only, more terms than one launch
or one buffer takes, memory that other buffers hold, and device waits that run out.
The oracle and dense diagonalisation are the reference, FP64 to a relative 1e-10.
"""

import math
import threading

import numpy as np
import pytest
import scipy.sparse as sp

import tbplas_b200 as tb
from tbplas_b200 import _native as nat
from tbplas_b200.fortran import f2py
from oracle import oracle

from conftest import bessel_series, rel_err, unit_states

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _backend():
    f2py.set_backend(precision="fp64", batch=16, device=0, state_kind="exp", term_kernel=0,
                     use_graphs=True, vector_width=0, threads_per_block=0, rows_per_tile=0)
    yield
    f2py.set_backend(precision="fp64", batch=16, term_kernel=0, vector_width=0)


@pytest.mark.parametrize("n_t", [20, 80])
def test_coupled_realisations(n_t):
    """A matrix that couples the row ranges: each range's part of <psi(0)|psi(t)> on the
    time-stepped route below and above 64 steps, and the norm check still refuses it."""
    s = tb.make_graphene_sample(5, 4, disorder=1.0, rescale=9.0, seed=5)
    h = s.build_ham_csr()
    off = [0, 13, h.shape[0]]
    bes = bessel_series(math.pi)
    args = (bes, h.indptr, h.indices, h.data, off, 2, 11, n_t)
    _, per = f2py.tbpm_dos_segmented(*args, 10 ** 6, 1e-9, per_state=True)
    e, v = np.linalg.eigh(h.toarray())
    for b in range(2):
        parts = [oracle.random_state(off[k + 1] - off[k], 11 * (2 * k + b + 1)) for k in range(2)]
        w = np.concatenate([p / np.linalg.norm(p) for p in parts])
        wt = np.exp(-1j * math.pi * np.outer(e, np.arange(n_t + 1))) * (v.conj().T @ w)[:, None]
        terms = w.conj()[:, None] * (v @ wt)
        assert rel_err(per[:, b], [terms[:13].sum(0), terms[13:].sum(0)]) < 1e-10
    with pytest.raises(nat.NormError):
        f2py.tbpm_dos_segmented(*args, 16, 1e-9)


def _lossy(eps):
    """A sample with -i eps on every site: the states decay by exp(-eps tau t)."""
    h = tb.make_graphene_sample(3, 2, disorder=1.0, rescale=9.0, seed=5).build_ham_csr()
    h = sp.csr_matrix(h - 1j * eps * sp.identity(h.shape[0]))
    h.sort_indices()
    return h


def test_loss_below_the_hermiticity_tolerance_reaches_the_norm_check():
    """2 eps tau t = 2.9e-11 at the check, the threshold is 1e-11."""
    h = _lossy(9e-15)
    wf0 = unit_states(1, h.shape[0], seed=1)
    bes = bessel_series(math.pi)
    with pytest.raises(nat.NormError):
        f2py.tbpm_dos_states(bes, h.indptr, h.indices, h.data, wf0, 512, 512, 1e-11)
    f2py.tbpm_dos_states(bes, h.indptr, h.indices, h.data, wf0, 512, 512, 1e-9)


@pytest.mark.parametrize("n_t", [300, 16384])
def test_loss_below_the_hermiticity_tolerance_over_long_runs(n_t):
    """The decay grows with the run: 8e-12 and 4.6e-10 at its end."""
    h = _lossy(9e-15)
    wf0 = unit_states(1, h.shape[0], seed=1)
    bes = bessel_series(math.pi)
    got = f2py.tbpm_dos_states(bes, h.indptr, h.indices, h.data, wf0, n_t, 10 ** 6, 1e-9)
    ref = oracle.tbpm_dos(bes, h.indptr, h.indices, h.data, n_t, wf0=wf0)
    assert rel_err(got, ref) < 1e-10


@pytest.mark.parametrize("prec,size,nx,n_t,tol", [("fp64", 2e-16, 3, 60000, 1e-9),
                                                  ("fp32", 3e-8, 20, 600, 3e-5)])
def test_conjugates_to_rounding_stay_on_the_short_route(prec, size, nx, n_t, tol):
    """Off-diagonal entries whose transposes differ by a rounding: a launch or less per
    step, not the 19 of time stepping; against the levels of the matrix without them
    (FP64: their own error, 4e-16 pi 60000 = 8e-11)."""
    s = tb.make_graphene_sample(nx, nx, disorder=1.0, rescale=9.0, seed=5)
    s.set_magnetic_field(60.0)
    h = s.build_ham_csr()
    rng = np.random.default_rng(2)
    off = h.indices != np.repeat(np.arange(h.shape[0]), np.diff(h.indptr))
    data = h.data * (1 + off * size * rng.choice([-1, 0, 1], h.data.size))
    wf0 = unit_states(1, h.shape[0], seed=1)
    f2py.set_backend(precision=prec)
    got = f2py.tbpm_dos_states(bessel_series(math.pi), h.indptr, h.indices, data, wf0, n_t, 128,
                               1e-9)
    assert f2py._ctx().last_stats()[0] < n_t
    e, v = np.linalg.eigh(h.toarray())
    w = abs(v.conj().T @ wf0[0]) ** 2
    ref = np.exp(-1j * math.pi * np.outer(np.arange(n_t + 1), e)) @ w
    assert rel_err(got, ref) < tol


@pytest.mark.parametrize("ns", [1, 2])
def test_packed_run_of_more_terms_than_a_grid_axis(ns):
    """50,000 steps of one tiny realisation: 75,000 terms whose sums are reduced
    together, where a grid has 65,535 blocks on its second axis."""
    h = tb.make_graphene_sample(2, 2, disorder=1.0, rescale=8.7, seed=3).build_ham_csr()
    bes = bessel_series(math.pi)
    _, per = f2py.tbpm_dos_segmented(bes, h.indptr, h.indices, h.data, [0, h.shape[0]], ns, 11,
                                     50000, 128, 1e-9, per_state=True)
    for b in range(ns):
        ref = oracle.tbpm_dos(bes, h.indptr, h.indices, h.data, 50000, seed=11 * (b + 1),
                              n_samples=1)
        assert rel_err(per[0, b], ref) < 1e-10


@pytest.mark.parametrize("nx,ns,n_t", [(40, 16, 8192), (16, 64, 16384)])
def test_memory_of_long_runs_is_bounded(nx, ns, n_t):
    """The one-launch and the cluster route in several launches (block partials of 450
    and 400 MB all together): the context grows by 64 MB of them, and the curve is the
    ring route's."""
    import torch
    h = tb.make_graphene_sample(nx, nx, disorder=1.0, rescale=9.0, seed=3).build_ham_csr()
    bes = bessel_series(math.pi)
    f2py.set_backend(batch=64)
    kept, nat._contexts = nat._contexts, {0: nat.Context(0)}
    try:
        def run(steps, states):
            return f2py.tbpm_dos(bes, h.indptr, h.indices, h.data, 7, steps, states, "", 0, 128,
                                 1e-9)
        run(2, 1)
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info(0)
        got = run(n_t, ns)
        used = free - torch.cuda.mem_get_info(0)[0]
        f2py.set_backend(term_kernel=2)
        assert rel_err(got, run(n_t, ns)) < 1e-10
        assert used < 200e6
    finally:
        nat._contexts[0].close()
        nat._contexts = kept


def test_buffers_of_an_earlier_call_are_not_free_memory():
    """Vectors of 1.07 GB held from a larger call and 0.13 GB free: several steps per
    expansion (1.4 GB) do not fit, although 3.3 GB are free or held together."""
    import torch
    s = tb.make_graphene_sample(192, 192, disorder=1.0, rescale=9.0, seed=2)
    ip, ix, hv, dx, dy = s.build_ham_dxy()
    bes = bessel_series(math.pi / 2)
    args = (bes, 40.0, 0.0, ip, ix, hv, s.rescale, dx, dy, 3, 64, 8, 2 ** 12, 1e-12, "", 0, 128,
            1e-9)
    want = f2py.tbpm_accond(*args)
    big = tb.make_graphene_device_sample(1024, 512, rescale=9.0, seed=2).build_ham_csr()
    kept, nat._contexts = nat._contexts, {0: nat.Context(0)}
    hold = None
    try:
        f2py.set_backend(batch=64)
        f2py.tbpm_dos(bes, big.indptr, big.indices, big.data, 7, 2, 64, "", 0, 128, 1e-9)
        f2py.set_backend(batch=16)
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info(0)
        hold = torch.empty(free - (128 << 20), dtype=torch.uint8, device="cuda")
        assert rel_err(f2py.tbpm_accond(*args), want) < 1e-12
    finally:
        del hold
        torch.cuda.empty_cache()
        nat._contexts[0].close()
        nat._contexts = kept


@pytest.mark.parametrize("kernel", [0, 1])
def test_grid_barrier_gives_up_and_the_context_stays_usable(kernel):
    """A grid barrier that one arrival never reaches: a time-out error, and the next
    run on the context is right."""
    ctx = f2py._ctx()
    with pytest.raises(nat.DeviceTimeoutError):
        ctx.call("tbpm_selftest_grid_wait", kernel, 1)
    h = tb.make_graphene_sample(8, 9, disorder=1.0, rescale=9.0, seed=4).build_ham_csr()
    wf0 = unit_states(2, h.shape[0], seed=9)
    bes = bessel_series(math.pi)
    got = f2py.tbpm_dos_states(bes, h.indptr, h.indices, h.data, wf0, 70, 64, 1e-9)
    ref = oracle.tbpm_dos(bes, h.indptr, h.indices, h.data, 70, wf0=wf0)
    assert rel_err(got, ref) < 1e-10
    with pytest.raises(ValueError):
        ctx.call("tbpm_selftest_grid_wait", 2, 1)


@pytest.mark.parametrize("n_t", [20, 70])
def test_eigenstates_without_a_norm_check_report_a_wait_that_ran_out(n_t):
    """Time-stepped and filtered quasi-eigenstates whose check step lies past the run."""
    s = tb.make_graphene_sample(8, 9, disorder=1.0, rescale=9.0, seed=4)
    h = s.build_ham_csr()
    wf0 = unit_states(2, h.shape[0], seed=9)
    t_step = 2 * math.pi / s.energy_range
    args = (bessel_series(math.pi), h.indptr, h.indices, h.data)
    energies = np.array([-0.4, 0.1, 0.3])
    f2py._ctx().call("tbpm_selftest_grid_wait", 0, 0)
    with pytest.raises(nat.DeviceTimeoutError):
        f2py.tbpm_eigenstates_states(*args, wf0, n_t, t_step, energies, 128, 1e-9)
    got = f2py.tbpm_eigenstates_states(*args, wf0, n_t, t_step, energies, 128, 1e-9)
    ref = oracle.tbpm_eigenstates(*args, n_t, t_step, energies, wf0=wf0)
    assert rel_err(got, ref) < 1e-10


def test_norm_check_refuses_moments_that_no_state_has():
    """The sums of a state with three levels give its curve; with one of them beyond the
    state's norm, or not a number, the norm check refuses the run."""
    x, w, n_t = np.array([-0.9, 0.2, 0.7]), np.array([0.5, 0.2, 0.3]), 80
    bes = np.array(bessel_series(math.pi))
    k = np.arange(200)
    t = np.cos(k[:, None] * np.arccos(x))
    sums = np.stack([(w * t[1:] ** 2).sum(1), (w * t[1:] * t[:-1]).sum(1)], 1)
    corr = np.zeros(n_t + 1, dtype=complex)
    f2py.set_backend(precision="fp64")
    f2py.tbpm_dos([1.0, 0.1, 0.01], [0, 0], [], [], 1, 1, 1, "", 0, 128, 1e-9)  # FP64 resident

    def run(s):
        f2py._ctx().call("tbpm_selftest_moments", nat.ptr(bes), bes.size, nat.ptr(s), len(s), n_t,
                         nat.ptr(corr))
    run(sums)
    ref = (w * np.exp(-1j * math.pi * x * np.arange(n_t + 1)[:, None])).sum(1)
    assert rel_err(corr, ref) < 1e-12
    for row, col, value, err in ((120, 0, 1.0 + 1e-6, nat.NormError),
                                 (33, 1, -1.1, nat.NormError), (150, 0, 1e30, nat.NormError),
                                 (7, 1, np.nan, nat.NanError)):
        bad = sums.copy()
        bad[row, col] = value
        with pytest.raises(err):
            run(bad)


def test_contexts_in_several_threads():
    """Twelve threads, each with its own context and a block shape of its own (launches
    of one kernel with different shared memory): every call returns the thread's first
    result bit for bit."""
    bes = nat.as_c(bessel_series(math.pi), np.float64)
    failed = []

    def work(nx):
        h = tb.make_graphene_sample(nx, 100, disorder=1.0, rescale=9.0, seed=2).build_ham_csr()
        ip, ix = nat.as_c(h.indptr, np.int32), nat.as_c(h.indices, np.int32)
        hv = nat.as_c(h.data, np.complex128)
        ctx = nat.Context(0)
        first = None
        try:
            for _ in range(500):
                corr = np.zeros(65, dtype=np.complex128)
                ctx.call("tbpm_dos", nat.ptr(bes), bes.size, nat.ptr(ip), nat.ptr(ix), nat.ptr(hv),
                         ip.size - 1, hv.size, 7, 64, 1, 0, 128, 1e-9, nat.ptr(corr))
                first = corr if first is None else first
                if not np.array_equal(first, corr):
                    failed.append((nx, rel_err(corr, first)))
        except nat.TbpmError as e:
            failed.append((nx, str(e)))
        finally:
            ctx.close()

    threads = [threading.Thread(target=work, args=(40 + 2 * i,)) for i in range(12)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


@pytest.fixture(scope="module")
def sample():
    s = tb.make_graphene_sample(9, 11, disorder=1.0, rescale=9.0, seed=21)
    s.set_magnetic_field(30.0)
    return s


KERNELS = pytest.mark.parametrize("kernel", [1, 2])  # grid-stride, ring: a launch per term
PRECS = pytest.mark.parametrize("prec", ["fp64", "fp32"])


@KERNELS
@PRECS
def test_eigenstates_by_launched_terms(sample, kernel, prec):
    h = sample.build_ham_csr()
    wf = unit_states(3, h.shape[0], seed=6)
    t_step = 2 * math.pi / sample.energy_range
    energies = np.linspace(-2.0, 2.0, 9) + 0.01
    args = (bessel_series(math.pi), h.indptr, h.indices, h.data)
    f2py.set_backend(precision=prec, term_kernel=kernel)
    got = f2py.tbpm_eigenstates_states(*args, wf, 97, t_step, energies, 64, 1e-9)
    ref = oracle.tbpm_eigenstates(*args, 97, t_step, energies, wf0=wf)
    assert rel_err(got, ref) < {"fp64": 1e-10, "fp32": 5e-5}[prec]


@KERNELS
@PRECS
def test_ac_and_polarisation_by_launched_terms(sample, kernel, prec):
    """Expansions of 57 (FP32: 36) vectors in windows of 32: several window borders."""
    ip, ix, hv, dx, dy = sample.build_ham_dxy()
    h = sample.build_ham_csr()
    wf = unit_states(3, h.shape[0], seed=21)
    bes = bessel_series(math.pi / 2)
    beta = sample.rescale / (tb.KB * 3000.0)
    f2py.set_backend(precision=prec, term_kernel=kernel)
    tol = {"fp64": 1e-10, "fp32": 2e-5}[prec]
    args = (bes, beta, 0.05, ip, ix, hv, sample.rescale, dx, dy)
    got = f2py.tbpm_accond_states(*args, wf, 90, 2 ** 15, 1e-12, 64, 1e-9)
    assert rel_err(got, oracle.tbpm_accond(*args, 90, wf0=wf)) < tol
    q = [[1.3, 0.2, 0.0], [0.0, 2.0, 0.0]]
    args = (bes, beta, 0.0, h.indptr, h.indices, h.data, *sample.orb_pos.T.copy(), q)
    got = f2py.tbpm_dyn_pol_states(*args, wf, 90, 2 ** 15, 1e-12, 64, 1e-9)
    assert rel_err(got, oracle.tbpm_dyn_pol(*args, 90, wf0=wf)) < tol


@pytest.mark.parametrize("kernel", [0, 1, 2])
@PRECS
def test_dc_by_launched_terms(sample, kernel, prec):
    """Energies inside the populated spectrum.  FP32: a recurrence of M = 280 terms loses
    at most 7 M rounding errors of 6e-8, 1.2e-4, and a value divides by |<wf0|QE>|, which
    is above a quarter of |QE| there."""
    ip, ix, hv, dx, dy = sample.build_ham_dxy()
    wf0 = unit_states(3, ip.size - 1, seed=31)
    n_t = 89
    e = np.array([0.5 * i * sample.energy_range / n_t - sample.energy_range / 2.
                  for i in range(2 * n_t)])
    sel = np.where((e >= 1.0) & (e <= 3.0))[0]
    t_step = 2 * math.pi / sample.energy_range
    args = (bessel_series(math.pi), ip, ix, hv, sample.rescale, dx, dy)
    f2py.set_backend(precision=prec, term_kernel=kernel)
    got = f2py.tbpm_dccond_states(*args, wf0, n_t, t_step, e, sel, 60, 1e-9)
    ref = oracle.tbpm_dccond(*args, n_t, t_step, e, sel, wf0=wf0)
    assert rel_err(got[0], ref[0]) < {"fp64": 1e-10, "fp32": 3e-5}[prec]
    assert rel_err(got[1], ref[1]) < {"fp64": 1e-10, "fp32": 5e-4}[prec]


@KERNELS
def test_dc_block_partials_in_several_reductions(kernel):
    """32 states of 5000 orbitals: the launched terms' block partials are reduced in
    several chunks of 64 MB, those of the one-launch route window by window."""
    s = tb.make_graphene_sample(50, 50, disorder=1.0, rescale=9.0, seed=3)
    ip, ix, hv, dx, dy = s.build_ham_dxy()
    bes = bessel_series(math.pi)
    energies, sel = np.array([1.5, 2.0]), np.arange(2)
    out = []
    for k in (0, kernel):
        f2py.set_backend(batch=32, term_kernel=k)
        out.append(f2py.tbpm_dccond(bes, 40.0, 0.0, ip, ix, hv, s.rescale, dx, dy, 5, 300, 32,
                                    math.pi / s.rescale, energies, sel, "", "", 0, 128, 1e-9))
    assert rel_err(out[1][0], out[0][0]) < 1e-12
    assert rel_err(out[1][1], out[0][1]) < 1e-10


@pytest.mark.parametrize("n", [150, 221])
def test_dc_of_general_matrices_inside_the_spectrum(n):
    """Rows of no entry up to twelve, unsorted columns, energies where the levels lie."""
    rng = np.random.default_rng(n)
    m = sp.random(n, n, density=3.0 / n, random_state=rng, format="csr")
    m = m + 1j * sp.random(n, n, density=3.0 / n, random_state=rng, format="csr")
    m = sp.csr_matrix(m + m.conj().T)
    m = sp.csr_matrix(m * (0.9 / abs(m).sum(1).max()))
    pos = rng.standard_normal((2, n))
    rows = np.repeat(np.arange(n), np.diff(m.indptr))
    dx, dy = pos[:, m.indices] - pos[:, rows]
    wf0 = unit_states(3, n, seed=21)
    levels = np.linalg.eigvalsh(m.toarray())
    energies, sel = np.quantile(levels, [0.2, 0.4, 0.6, 0.8]), np.arange(4)
    args = (bessel_series(math.pi), m.indptr, m.indices, m.data, 1.0, dx, dy)
    got = f2py.tbpm_dccond_states(*args, wf0, 70, math.pi, energies, sel, 64, 1e-9)
    ref = oracle.tbpm_dccond(*args, 70, math.pi, energies, sel, wf0=wf0)
    assert rel_err(got[0], ref[0]) < 1e-10
    assert rel_err(got[1], ref[1]) < 1e-10


@pytest.mark.parametrize("driver", ["ac", "dc", "psi_t"])
def test_driver_calls_end_a_session(sample, driver):
    """A driver's call takes the vectors over (and may give them back to the device): the
    session is over, not continued on what is left."""
    ip, ix, hv, dx, dy = sample.build_ham_dxy()
    bes = nat.as_c(bessel_series(math.pi), np.float64)
    wf = unit_states(2, ip.size - 1, seed=1)
    ctx = f2py._ctx()
    arrays = [nat.as_c(a, t) for a, t in ((ip, np.int32), (ix, np.int32), (hv, np.complex128),
                                          (dx, np.float64), (dy, np.float64))]
    ctx.call("tbpm_ham_upload", *map(nat.ptr, arrays[:3]), ip.size - 1, ix.size,
             *map(nat.ptr, arrays[3:]), sample.rescale)
    ctx.call("tbpm_session_dos_begin", nat.ptr(bes), bes.size, 4, 7, 0, 4, 40)
    ctx.call("tbpm_session_advance", 4)

    class Uploaded:  # calls with this in the place of indptr run on the uploaded Hamiltonian
        @staticmethod
        def make_resident(_):
            return ip.size - 1, ix.size
    args = (bes, Uploaded, None, None)
    if driver == "ac":
        f2py.tbpm_accond_states(bes, 8.0, 0.0, *args[1:], sample.rescale, None, None, wf, 64,
                                2 ** 12, 1e-12, 128, 1e-9)
    elif driver == "dc":
        f2py.tbpm_eigenstates_states(*args, wf, 64, 0.3, [0.1], 128, 1e-9)
    else:
        f2py.tbpm_psi_t(*args, wf[0], np.array([0, 64]), 64, 128, 1e-9)
    with pytest.raises(nat.TbpmError):
        ctx.call("tbpm_session_advance", 4)


def _launches():
    return f2py._ctx().last_stats()[0]


@pytest.mark.parametrize("n_en,filtered", [(4, True), (1000, False)])
def test_long_runs_whose_filters_cost_more_than_the_steps(sample, n_en, filtered):
    """8192 steps: a few energies by filters (a vector per 0.33 steps), 1000 of them time-stepped
    as a transform of 25,000 x 25,000 x 1000 products would take longer; both routes' densities
    at the energies they share agree."""
    h = sample.build_ham_csr()
    wf = unit_states(1, h.shape[0], seed=6)
    energies = np.linspace(-2.0, 2.0, n_en) + 0.003
    t_step = 2 * math.pi / sample.energy_range
    args = (bessel_series(math.pi), h.indptr, h.indices, h.data, wf, 8192, t_step)
    got = f2py.tbpm_eigenstates_states(*args, energies, 128, 1e-9)
    assert (_launches() < 8192) == filtered
    if not filtered:
        pick = [0, 333, 999]
        few = f2py.tbpm_eigenstates_states(*args, energies[pick], 128, 1e-9)
        assert _launches() < 8192
        assert rel_err(got[pick], few) < 1e-8


def test_dc_with_stepped_quasi_eigenstates_and_expanded_currents(sample):
    """The same choice in tbpm_dccond: phase 1 time-stepped (its filters would cost more),
    phase 2 by several steps per expansion, against both phases of the short route."""
    ip, ix, hv, dx, dy = sample.build_ham_dxy()
    wf = unit_states(2, ip.size - 1, seed=6)
    energies = np.linspace(1.0, 3.0, 1000)
    t_step = 2 * math.pi / sample.energy_range
    args = (bessel_series(math.pi), ip, ix, hv, sample.rescale, dx, dy, wf, 6000, t_step, energies)
    dos, dc = f2py.tbpm_dccond_states(*args, np.arange(1000), 128, 1e-9)
    stepped = _launches()
    pick = np.array([0, 500, 999])
    dos3, dc3 = f2py.tbpm_dccond_states(*args, pick, 128, 1e-9)
    assert _launches() < 6000 * 4 < 6000 * 19 < stepped < 6000 * 26
    assert rel_err(dos, dos3) < 1e-10
    assert rel_err(dc[:, pick], dc3[:, :3]) < 1e-8


def test_dos_of_a_large_time_step_over_a_long_run(sample):
    """Twelve times the usual time step, 60,000 steps: two million moments would cost more than
    the products they save; 2000 steps take the moments."""
    h = sample.build_ham_csr()
    wf = unit_states(1, h.shape[0], seed=6)
    bes = bessel_series(12 * math.pi)
    e, v = np.linalg.eigh(h.toarray())
    w = abs(v.conj().T @ wf[0]) ** 2
    for n_t, moments in ((2000, True), (60000, False)):
        got = f2py.tbpm_dos_states(bes, h.indptr, h.indices, h.data, wf, n_t, 128, 1e-9)
        assert (_launches() < n_t) == moments
        ref = np.exp(-12j * math.pi * np.outer(np.arange(n_t + 1), e)) @ w
        assert rel_err(got, ref) < 1e-8

"""GPU check (cuFFT) against the reference's checkcode: the goldens hold the fit
and Coulomb errors the reference printed for its own theta; the GPU check run
on that same theta must reproduce them. Also the check inside ISDF(), and the
sampled-pair check (isdf_check_sampled) that reaches sizes the full check
refuses."""
import numpy as np
import pytest

from conftest import load_golden, record_parity
from oracle import check as ocheck

import libisdf_b200 as isdf
from libisdf_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["small_s1s2", "small_mu0"])
def test_check_reproduces_reference_numbers(torch_cuda, name):
    torch = torch_cuda
    g = load_golden(name)
    a = (int(g["nocc"]), int(g["nv1"]), int(g["nc1"]), int(g["nv2"]), int(g["nc2"]))
    rk = int(g["rk_eff"])
    dom = isdf.Domain(length=tuple(g["length"]), num_grid=tuple(int(x) for x in g["ng"]))
    d_psi = torch.from_numpy(np.ascontiguousarray(g["psi"].T)).cuda()
    d_th = torch.from_numpy(np.ascontiguousarray(g["theta"].T)).cuda()
    th_before = d_th.clone()
    fe, ce = isdf.check(dom, d_psi, a[0], g["psi"].shape[1], *a[1:], rk, g["piv"], d_th)
    assert torch.equal(d_th, th_before)  # theta is read only
    assert abs(fe / float(g["fit_err"]) - 1) < 1e-9
    # the Coulomb error is a small difference of large sums: 1e-6 relative
    assert abs(ce / float(g["coul_err"]) - 1) < 1e-6


def test_check_inside_isdf_si8(torch_cuda):
    """Si8-like shape (40^3 grid, 32 states, mu = 320), check = true: the
    report carries both errors, equal to the numpy restatement's on the same
    theta."""
    torch = torch_cuda
    s = synth.SI8
    psi = synth.shape_orbitals(s, 0)
    dom = isdf.Domain(length=(s.length,) * 3, num_grid=(s.n,) * 3)
    d_psi = torch.from_numpy(np.ascontiguousarray(psi.T)).cuda()
    d_theta = torch.empty((s.mu, s.ng), dtype=torch.float64, device="cuda")
    piv = np.zeros(s.ng, dtype=np.int32)
    rep = isdf.ISDF(d_psi, dom, s.nocc, s.nstate, s.nv1, s.nc1, s.nv2, s.nc2, s.mu, d_theta, piv,
                    s.kmeans_iters, check=True)
    th = np.asfortranarray(d_theta.cpu().numpy().T)
    fe, ce = ocheck.check(psi, (s.n,) * 3, (s.length,) * 3, s.nocc, s.nv1, s.nc1, s.nv2, s.nc2,
                          rep.rk_eff, piv, th)
    assert rep.fit_err > 0 and rep.coul_err > 0
    assert abs(rep.fit_err / fe - 1) < 1e-8
    assert abs(rep.coul_err / ce - 1) < 1e-6


def _close(x, y, rel):
    return abs(x - y) <= rel * abs(y) + 1e-15


@pytest.mark.parametrize("name", ["small_s1s2", "small_mu0"])
def test_sampled_check_all_pairs_equals_full_check(torch_cuda, name):
    """The sampled check given every pair reproduces the full check (and so
    the reference's printed numbers); on a subset it equals the oracle's
    restatement with the reference's c^T Re(zeta^H V zeta) c form."""
    torch = torch_cuda
    g = load_golden(name)
    a = (int(g["nocc"]), int(g["nv1"]), int(g["nc1"]), int(g["nv2"]), int(g["nc2"]))
    rk = int(g["rk_eff"])
    ng, ln = tuple(int(x) for x in g["ng"]), tuple(g["length"])
    dom = isdf.Domain(length=ln, num_grid=ng)
    d_psi = torch.from_numpy(np.ascontiguousarray(g["psi"].T)).cuda()
    d_th = torch.from_numpy(np.ascontiguousarray(g["theta"].T)).cuda()
    npair = (a[1] + a[2]) * (a[3] + a[4])
    full = isdf.check(dom, d_psi, a[0], g["psi"].shape[1], *a[1:], rk, g["piv"], d_th)
    every = isdf.check_sampled(dom, d_psi, a[0], g["psi"].shape[1], *a[1:], rk, g["piv"], d_th,
                               np.arange(npair))
    assert _close(every[0], full[0], 1e-10) and _close(every[1], full[1], 1e-7)
    sub = np.random.default_rng(0).choice(npair, size=npair // 3, replace=False)
    got = isdf.check_sampled(dom, d_psi, a[0], g["psi"].shape[1], *a[1:], rk, g["piv"], d_th, sub)
    want = ocheck.check_sampled(g["psi"], ng, ln, *a, rk, g["piv"], g["theta"], sub)
    record_parity(f"sampled check {name}", "fit / Coulomb error (GPU; oracle)",
                  f"{got[0]:.6e} / {got[1]:.6e}; {want[0]:.6e} / {want[1]:.6e}")
    assert _close(got[0], want[0], 1e-9) and _close(got[1], want[1], 1e-6)


def test_sampled_check_at_si64(torch_cuda):
    """The check at a size the full check refuses: the Si64-like shape (80^3,
    256 states, 65536 pairs, mu = 2048 from K-means), 192 sampled pairs,
    against the oracle's restatement of the same pair block (fitted-density
    spectra; numpy FFT) on the same theta."""
    torch = torch_cuda
    s = synth.SI64
    psi = synth.shape_orbitals(s, 1, device="cuda")
    dom = isdf.Domain(length=(s.length,) * 3, num_grid=(s.n,) * 3)
    d_psi = torch.from_numpy(np.ascontiguousarray(psi.T)).cuda()
    d_theta = torch.empty((s.mu, s.ng), dtype=torch.float64, device="cuda")
    piv = np.zeros(s.ng, dtype=np.int32)
    rep = isdf.ISDF(d_psi, dom, s.nocc, s.nstate, s.nv1, s.nc1, s.nv2, s.nc2, s.mu, d_theta, piv,
                    s.kmeans_iters)
    with pytest.raises(isdf.IsdfError):
        isdf.check(dom, d_psi, s.nocc, s.nstate, s.nv1, s.nc1, s.nv2, s.nc2, rep.rk_eff, piv,
                   d_theta)
    npair = (s.nv1 + s.nc1) * (s.nv2 + s.nc2)
    pairs = np.sort(np.random.default_rng(1).choice(npair, size=192, replace=False))
    got = isdf.check_sampled(dom, d_psi, s.nocc, s.nstate, s.nv1, s.nc1, s.nv2, s.nc2,
                             rep.rk_eff, piv, d_theta, pairs)
    th = np.asfortranarray(d_theta[:rep.rk_eff].cpu().numpy().T)
    want = ocheck.check_sampled(psi, (s.n,) * 3, (s.length,) * 3, s.nocc, s.nv1, s.nc1, s.nv2,
                                s.nc2, rep.rk_eff, piv, th, pairs, fitted_spectra=True)
    record_parity("sampled check Si64", "fit / Coulomb error (GPU; oracle)",
                  f"{got[0]:.6e} / {got[1]:.6e}; {want[0]:.6e} / {want[1]:.6e}")
    assert _close(got[0], want[0], 1e-9) and _close(got[1], want[1], 1e-6)


@pytest.mark.parametrize("name", ["small_s1s2", "si8_example"])
def test_coulomb_matrix_matches_oracle(torch_cuda, name):
    """The ISDF Coulomb matrix Re(zeta^H V zeta) of theta, the quantity the
    reference's check forms at checkcode.cpp:249-288, against its numpy
    restatement (full complex spectra) on the reference's own theta."""
    torch = torch_cuda
    g = load_golden(name)
    rk = int(g["rk_eff"])
    ng, ln = tuple(int(x) for x in g["ng"]), tuple(g["length"])
    th = g["theta"] if "theta" in g else None
    if th is None:  # the Si8 example keeps only a few theta columns: refit on the GPU
        a = (int(g["nocc"]), int(g["nv1"]), int(g["nc1"]), int(g["nv2"]), int(g["nc2"]))
        d_psi = torch.from_numpy(np.ascontiguousarray(g["psi"].T)).cuda()
        d_th = torch.zeros((rk, g["psi"].shape[0]), dtype=torch.float64, device="cuda")
        isdf.fit(d_psi, g["psi"].shape[0], g["psi"].shape[1], *a, rk, g["piv"], d_th)
        th = np.asfortranarray(d_th.cpu().numpy().T)
    d_th = torch.from_numpy(np.ascontiguousarray(th.T)).cuda()
    d_A = torch.zeros((rk, rk), dtype=torch.float64, device="cuda")
    isdf.coulomb_matrix(isdf.Domain(length=ln, num_grid=ng), d_th, rk, d_A)
    A = d_A.cpu().numpy().T  # column-major rk x rk
    A_o = ocheck.coulomb_matrix(th, ng, ln, rk)
    err = float(np.linalg.norm(A - A_o) / np.linalg.norm(A_o))
    record_parity(f"Coulomb matrix {name}", "relative difference vs oracle", err, 1e-10)
    assert err <= 1e-10
    assert np.allclose(A, A.T, rtol=0, atol=1e-12 * np.abs(A).max())


@pytest.mark.parametrize("rk", [1, 2, 63, 64, 65, 130, 321])
@pytest.mark.parametrize("ng", [(14, 12, 10), (9, 15, 25)])
def test_coulomb_matrix_tile_edges(torch_cuda, rk, ng):
    """Around the 64-wide tiles of the symmetric product, odd and even sizes,
    depths that split unevenly. The product sums 2 nh terms: its rounding is at
    most that many half ulps of the norms."""
    torch = torch_cuda
    ln = (7.0, 8.0, 9.0)
    n = ng[0] * ng[1] * ng[2]
    th = np.asfortranarray(np.random.default_rng(rk).standard_normal((n, rk)))
    d_th = torch.from_numpy(np.ascontiguousarray(th.T)).cuda()
    d_A = torch.full((rk, rk), float("nan"), dtype=torch.float64, device="cuda")
    isdf.coulomb_matrix(isdf.Domain(length=ln, num_grid=ng), d_th, rk, d_A)
    torch.cuda.synchronize()
    A, A_o = d_A.cpu().numpy().T, ocheck.coulomb_matrix(th, ng, ln, rk)
    tol = 2 * (ng[0] // 2 + 1) * ng[1] * ng[2] * 2.0 ** -53
    assert np.linalg.norm(A - A_o) <= tol * np.linalg.norm(A_o)
    assert np.array_equal(A, A.T)


@pytest.mark.parametrize("ng", [(16, 12, 10), (9, 15, 25), (7, 7, 13)])
def test_coulomb_matrix_leaves_theta(torch_cuda, ng):
    """theta is the caller's: whole batches are transformed from it in place of a
    copy, the rest through one, aligned columns or not; it must come back as it
    was, and the result agree with the oracle's."""
    torch = torch_cuda
    rk, n = 300, ng[0] * ng[1] * ng[2]
    th = np.asfortranarray(np.random.default_rng(1).standard_normal((n, rk)))
    d_th = torch.from_numpy(np.ascontiguousarray(th.T)).cuda()
    before = d_th.clone()
    d_A = torch.empty((rk, rk), dtype=torch.float64, device="cuda")
    ln = (7.0, 8.0, 9.0)
    isdf.coulomb_matrix(isdf.Domain(length=ln, num_grid=ng), d_th, rk, d_A)
    torch.cuda.synchronize()
    assert torch.equal(d_th, before)
    A_o = ocheck.coulomb_matrix(th, ng, ln, rk)
    tol = 2 * (ng[0] // 2 + 1) * ng[1] * ng[2] * 2.0 ** -53
    assert np.linalg.norm(d_A.cpu().numpy().T - A_o) <= tol * np.linalg.norm(A_o)


def test_coulomb_matrix_kept_plans(torch_cuda):
    """More grids in turn than plans are kept, twice over, with the workspace
    released in between and from two threads: the same results each time."""
    import threading

    torch = torch_cuda
    rk, ln = 5, (7.0, 8.0, 9.0)
    grids = [(8, 6, 4), (9, 6, 4), (8, 7, 4), (8, 6, 5), (10, 6, 4), (4, 6, 8)]
    ths = [np.asfortranarray(np.random.default_rng(k).standard_normal((g[0] * g[1] * g[2], rk)))
           for k, g in enumerate(grids)]
    want = [ocheck.coulomb_matrix(t, g, ln, rk) for t, g in zip(ths, grids)]
    lib = isdf.lib()

    def run(fail):
        try:
            st = torch.cuda.Stream()
            for rep in range(2):
                for t, g, w in zip(ths, grids, want):
                    d_th = torch.from_numpy(np.ascontiguousarray(t.T)).cuda()
                    d_A = torch.empty((rk, rk), dtype=torch.float64, device="cuda")
                    torch.cuda.synchronize()
                    with lock:  # one workspace: calls on different streams in turn
                        isdf.coulomb_matrix(isdf.Domain(length=ln, num_grid=g), d_th, rk, d_A,
                                            stream=st.cuda_stream)
                        torch.cuda.synchronize()
                    a = d_A.cpu().numpy().T
                    if not np.linalg.norm(a - w) <= 1e-12 * np.linalg.norm(w):
                        fail.append((rep, g))
        except Exception as e:  # noqa: BLE001 - reported by the assertion below
            fail.append(repr(e))

    lock = threading.Lock()
    fail = []
    run(fail)
    lib.isdf_release_workspace()
    threads = [threading.Thread(target=run, args=(fail,)) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not fail


@pytest.mark.parametrize("own", [False, True])
def test_coulomb_matrix_is_done_on_return(torch_cuda, own):
    """Calls back to back, on the library's stream or on two of the caller's, and a
    fit behind one, all in the same workspace: every result may be read at once, and
    none is overwritten by the next call's scratch. The same bits as a call alone."""
    torch = torch_cuda
    grid, rk, ns = (40, 40, 40), 600, 40
    n, dom = 64000, isdf.Domain(length=(7.0, 8.0, 9.0), num_grid=grid)
    gen = torch.Generator(device="cuda").manual_seed(1)
    ths = [torch.randn((rk, n), dtype=torch.float64, device="cuda", generator=gen)
           for _ in range(2)]
    psi = torch.randn((ns, n), dtype=torch.float64, device="cuda", generator=gen)
    piv = np.arange(64, dtype=np.int32) * 997
    win = (ns // 2, ns // 2, ns // 2, ns // 2, ns // 2)
    streams = [torch.cuda.Stream().cuda_stream if own else 0 for _ in range(2)]

    def empty(*shape):
        return torch.full(shape, float("nan"), dtype=torch.float64, device="cuda")

    alone = []
    for th in ths:
        A = empty(rk, rk)
        torch.cuda.synchronize()
        isdf.coulomb_matrix(dom, th, rk, A, stream=streams[0])
        torch.cuda.synchronize()
        alone.append(A.cpu())
    fit_alone = empty(64, n)
    torch.cuda.synchronize()
    isdf.fit(psi, n, ns, *win, 64, piv, fit_alone, stream=streams[1])
    torch.cuda.synchronize()

    got, theta = [empty(rk, rk) for _ in ths], empty(64, n)
    torch.cuda.synchronize()
    for A, th, st in zip(got, ths, streams):
        isdf.coulomb_matrix(dom, th, rk, A, stream=st)
    host = [A.cpu() for A in got]  # on the current stream, which waits for neither
    assert all(torch.equal(h, w) for h, w in zip(host, alone))
    last = empty(rk, rk)
    torch.cuda.synchronize()
    isdf.coulomb_matrix(dom, ths[0], rk, last, stream=streams[0])
    isdf.fit(psi, n, ns, *win, 64, piv, theta, stream=streams[1])
    assert torch.equal(last.cpu(), alone[0])
    assert torch.equal(theta, fit_alone)

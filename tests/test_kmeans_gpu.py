"""K-means selection on the GPU against the reference (bit-exact weight, piv,
effective mu and iteration count)."""
import numpy as np
import pytest

from conftest import load_golden, record_parity
from oracle import port

import libisdf_b200 as isdf
from libisdf_b200 import synth

pytestmark = pytest.mark.gpu
CASES = ["si8_example", "small_s1s2", "small_mu0", "small_iters0", "small_early"]


def _dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(np.asfortranarray(a).T)).cuda()


@pytest.mark.parametrize("name", CASES)
def test_weight_bit_exact(torch_cuda, name):
    torch = torch_cuda
    g = load_golden(name)
    psi = g["psi"]
    d_psi = _dev(torch, psi)
    d_w = torch.empty(psi.shape[0], dtype=torch.float64, device="cuda")
    isdf.kmeans_weight(d_psi, psi.shape[0], psi.shape[1], int(g["nocc"]), int(g["nv1"]),
                       int(g["nc1"]), int(g["nv2"]), int(g["nc2"]), d_w)
    torch.cuda.synchronize()
    assert np.array_equal(d_w.cpu().numpy(), g["weight"])


@pytest.mark.parametrize("name", CASES)
def test_select_matches_reference(torch_cuda, name):
    torch = torch_cuda
    g = load_golden(name)
    dom = isdf.Domain(length=tuple(g["length"]), num_grid=tuple(int(x) for x in g["ng"]))
    d_w = torch.from_numpy(g["weight"]).cuda()
    piv, rk, it, npt = isdf.kmeans_select(dom, d_w, int(g["rk_requested"]), int(g["iters"]),
                                          rand_seed=int(g["rand_seed"]))
    assert (rk, it) == (int(g["rk_eff"]), int(g["n_iter"]))
    assert np.array_equal(piv, g["piv"])


def test_select_si8_synthetic_matches_oracle(torch_cuda):
    """Si8-like shape: 40^3 grid, 32 states, mu = 320, 100 iterations."""
    torch = torch_cuda
    s = synth.SI8
    psi = synth.shape_orbitals(s, 0)
    ng, ln = (s.n,) * 3, (s.length,) * 3
    piv_o, rk_o, it_o, w_o = port.kmeans_piv(psi, ng, ln, s.nocc, s.nv1, s.nc1, s.nv2, s.nc2,
                                             s.mu, s.kmeans_iters)
    g = load_golden("si8_synth_seed0")
    if synth.sha256(psi) == str(g["psi_sha256"]):  # same bits as when the golden was made
        assert np.array_equal(piv_o, g["piv"]) and rk_o == int(g["rk_eff"])
    dom = isdf.Domain(length=ln, num_grid=ng)
    d_psi = _dev(torch, psi)
    d_theta = torch.empty((s.mu, s.ng), dtype=torch.float64, device="cuda")
    piv = np.zeros(s.ng, dtype=np.int32)
    rep = isdf.ISDF(d_psi, dom, s.nocc, s.nstate, s.nv1, s.nc1, s.nv2, s.nc2, s.mu, d_theta, piv,
                    s.kmeans_iters)
    assert rep.rk_eff == rk_o and rep.kmeans_iters == it_o
    assert np.array_equal(piv, piv_o)
    # zero-filled columns past the effective mu
    assert float(d_theta[rep.rk_eff:].abs().max().cpu()) == 0.0 if rep.rk_eff < s.mu else True


def test_select_is_repeatable(torch_cuda):
    torch = torch_cuda
    g = load_golden("small_s1s2")
    dom = isdf.Domain(length=tuple(g["length"]), num_grid=tuple(int(x) for x in g["ng"]))
    d_w = torch.from_numpy(g["weight"]).cuda()
    a = isdf.kmeans_select(dom, d_w, 40, 50)
    b = isdf.kmeans_select(dom, d_w, 40, 50)
    assert np.array_equal(a[0], b[0]) and a[1:] == b[1:]


@pytest.mark.parametrize("seed", [0, 1])
def test_select_heavy_zero_tail(torch_cuda, seed):
    """Half of the grid falls below the weight filter, so half of the K-means
    points are copies of grid point 0 (the reference's zero-initialised index
    tail), here carrying the largest weight: their cluster's fold is dominated
    by that repeated addition."""
    torch = torch_cuda
    rng = np.random.default_rng(seed)
    ng = (20, 21, 19)
    n = int(np.prod(ng))
    w = rng.uniform(0.1, 1.0, size=n) ** 3
    w[rng.random(n) < 0.5] = 1e-13
    w[0] = 1.7
    length = (9.5, 10.0, 9.0)
    piv_o, rk_o, it_o = port.kmeans(w, ng, length, 50, 30)
    piv, rk, it, npt = isdf.kmeans_select(isdf.Domain(length=length, num_grid=ng),
                                          torch.from_numpy(w).cuda(), 50, 30)
    assert npt < n / 2 + n / 10
    assert (rk, it) == (rk_o, it_o)
    assert np.array_equal(piv, piv_o)


@pytest.mark.parametrize("mu,seed", [(500, 3), (1, 4), (2000, 5)])
def test_select_random_weights(torch_cuda, mu, seed):
    """Random weights on an anisotropic grid: many centroids per cell ring,
    equal-distance ties between lattice points, the pruned search against
    the brute-force restatement."""
    torch = torch_cuda
    rng = np.random.default_rng(seed)
    ng = (30, 25, 20)
    n = int(np.prod(ng))
    w = rng.uniform(0.0, 1.0, size=n) ** 4
    length = (12.0, 7.5, 9.0)
    piv_o, rk_o, it_o = port.kmeans(w, ng, length, mu, 40)
    piv, rk, it, npt = isdf.kmeans_select(isdf.Domain(length=length, num_grid=ng),
                                          torch.from_numpy(w).cuda(), mu, 40)
    assert (rk, it) == (rk_o, it_o)
    assert np.array_equal(piv, piv_o)


def _perturbed_prev(g, seed=1):
    """Pivots of a previous solve on a slightly different weight (as an SCF
    loop's last iteration would have left them)."""
    ng = tuple(int(x) for x in g["ng"])
    ln = tuple(float(x) for x in g["length"])
    rng = np.random.default_rng(seed)
    w2 = np.abs(g["weight"] * (1 + 0.05 * rng.standard_normal(g["weight"].shape)))
    prev, _, _ = port.kmeans(w2, ng, ln, int(g["rk_requested"]), int(g["iters"]))
    return prev


@pytest.mark.parametrize("name", ["si8_example", "small_s1s2", "small_mu0", "small_iters0"])
def test_warm_start_matches_reference(torch_cuda, name):
    """K-means warm start (utility.cpp:725-749) through ISDF() with
    kmeans_warm_start: the same piv, effective mu, iteration count and number
    of reused pivots as the port, and as the reference's own KMEAN called
    with the same previous piv where the reference build is present."""
    torch = torch_cuda
    g = load_golden(name)
    ng = tuple(int(x) for x in g["ng"])
    ln = tuple(float(x) for x in g["length"])
    a = (int(g["nocc"]), int(g["nv1"]), int(g["nc1"]), int(g["nv2"]), int(g["nc2"]))
    mu, iters = int(g["rk_requested"]), int(g["iters"])
    prev = _perturbed_prev(g)
    piv_o, rk_o, it_o, used_o = port.kmeans_warm(g["weight"], ng, ln, mu, iters, prev)
    from oracle import ref

    if ref.available():
        r = ref.kmeans_warm(g["weight"], ng, ln, mu, iters, prev)
        assert np.array_equal(r[0], piv_o) and r[1:] == (rk_o, it_o, used_o)
    psi = g["psi"]
    d_psi = _dev(torch, psi)
    d_theta = torch.empty((mu, psi.shape[0]), dtype=torch.float64, device="cuda")
    piv = prev.copy()
    rep = isdf.ISDF(d_psi, isdf.Domain(length=ln, num_grid=ng), a[0], psi.shape[1], *a[1:], mu,
                    d_theta, piv, iters, options=isdf.Options(kmeans_warm_start=True))
    assert (rep.rk_eff, rep.kmeans_iters, rep.kmeans_warm_pivots) == (rk_o, it_o, used_o)
    assert np.array_equal(piv, piv_o)
    # without the option the caller's piv is ignored, as in the reference
    piv = prev.copy()
    rep = isdf.ISDF(d_psi, isdf.Domain(length=ln, num_grid=ng), a[0], psi.shape[1], *a[1:], mu,
                    d_theta, piv, iters)
    assert rep.kmeans_warm_pivots == -1 and np.array_equal(piv, g["piv"])


def test_warm_start_si8_perturbed_orbitals(torch_cuda):
    """An SCF-like step on the Si8-like shape: the orbitals change slightly
    between two solves; the second solve starts from the first one's piv and
    equals the port's warm start bit for bit."""
    torch = torch_cuda
    s = synth.SI8
    psi = synth.shape_orbitals(s, 0)
    rng = np.random.default_rng(9)
    psi2 = np.asfortranarray(np.linalg.qr(psi + 1e-3 * rng.standard_normal(psi.shape))[0])
    ng, ln = (s.n,) * 3, (s.length,) * 3
    a = (s.nocc, s.nv1, s.nc1, s.nv2, s.nc2)
    dom = isdf.Domain(length=ln, num_grid=ng)
    d_theta = torch.empty((s.mu, s.ng), dtype=torch.float64, device="cuda")
    piv = np.zeros(s.ng, dtype=np.int32)
    rep1 = isdf.ISDF(_dev(torch, psi), dom, s.nocc, s.nstate, *a[1:], s.mu, d_theta, piv,
                     s.kmeans_iters)
    prev = piv.copy()
    w2 = port.weight(psi2, *a)
    piv_o, rk_o, it_o, used_o = port.kmeans_warm(w2, ng, ln, s.mu, s.kmeans_iters, prev)
    cold = port.kmeans(w2, ng, ln, s.mu, s.kmeans_iters)
    rep2 = isdf.ISDF(_dev(torch, psi2), dom, s.nocc, s.nstate, *a[1:], s.mu, d_theta, piv,
                     s.kmeans_iters, options=isdf.Options(kmeans_warm_start=True))
    assert (rep2.rk_eff, rep2.kmeans_iters, rep2.kmeans_warm_pivots) == (rk_o, it_o, used_o)
    assert np.array_equal(piv, piv_o)
    record_parity("K-means warm start Si8-like", "Lloyd iterations warm / cold",
                  f"{rep2.kmeans_iters} / {cold[2]} (first solve {rep1.kmeans_iters})")


def test_batched_selection_matches_reference(torch_cuda):
    """The batched selection of small systems (one cooperative launch, a CTA
    group per system, the serving loop's path for small requests): every
    result equals the reference's (goldens: piv, effective mu, iteration
    count, including the npt < mu early return) and, for the Si8-like system
    and a random-weight grid, the port's, in one batch of mixed sizes."""
    torch = torch_cuda
    names = ["si8_example", "small_s1s2", "small_mu0", "small_iters0", "small_early"]
    doms, ws, mus, its, want = [], [], [], [], []
    for name in names:
        g = load_golden(name)
        doms.append(isdf.Domain(length=tuple(g["length"]), num_grid=tuple(int(x) for x in g["ng"])))
        ws.append(torch.from_numpy(g["weight"]).cuda())
        mus.append(int(g["rk_requested"]))
        its.append(int(g["iters"]))
        want.append((g["piv"], int(g["rk_eff"]), int(g["n_iter"])))
    s = synth.SI8
    psi = synth.shape_orbitals(s, 0)
    w8 = port.weight(psi, s.nocc, s.nv1, s.nc1, s.nv2, s.nc2)
    p8, r8, i8 = port.kmeans(w8, (s.n,) * 3, (s.length,) * 3, s.mu, s.kmeans_iters)
    doms.append(isdf.Domain(length=(s.length,) * 3, num_grid=(s.n,) * 3))
    ws.append(torch.from_numpy(w8).cuda())
    mus.append(s.mu)
    its.append(s.kmeans_iters)
    want.append((p8, r8, i8))
    rng = np.random.default_rng(3)
    ng = (30, 25, 20)
    wr = rng.uniform(0.0, 1.0, size=int(np.prod(ng))) ** 4
    pr, rr, ir = port.kmeans(wr, ng, (12.0, 7.5, 9.0), 500, 40)
    doms.append(isdf.Domain(length=(12.0, 7.5, 9.0), num_grid=ng))
    ws.append(torch.from_numpy(wr).cuda())
    mus.append(500)
    its.append(40)
    want.append((pr, rr, ir))
    got = isdf.kmeans_select_batch(doms, ws, mus, its, rand_seed=1)
    for k, ((piv, rk, it, _), (wp, wr_, wi)) in enumerate(zip(got, want)):
        assert (rk, it) == (wr_, wi), k
        assert np.array_equal(piv, wp), k


@pytest.mark.parametrize("kind", ["ties", "binades", "flat", "plane"])
@pytest.mark.parametrize("length", [(20.0, 20.0, 20.0), (10.26, 9.7, 11.3)])
def test_select_long_folds_match_oracle(torch_cuda, kind, length):
    """Clusters of up to thousands of points, whose weighted sums must round as
    the one-by-one fold does: weights that tie with the sums' last place, that
    span the kept range, that are all equal, and points in one plane (sums of
    zeros); exact integer coordinates and rounded ones."""
    torch = torch_cuda
    ng = (20, 21, 1 if kind == "plane" else 20)
    n = ng[0] * ng[1] * ng[2]
    rng = np.random.default_rng(7)
    if kind == "ties":
        w = rng.integers(1, 1 << 12, n) * 2.0 ** rng.integers(-20, 0, n) + 2.0 ** -31
    elif kind == "binades":
        w = np.exp(rng.uniform(np.log(2e-8), 0.0, n))
    else:
        w = np.full(n, 0.7)
    w[rng.integers(0, n, n // 9)] = 0.0  # dropped by the filter: a zero tail
    w[0] = 0.3
    for mu in (3, 24):
        piv_o, rk_o, it_o = port.kmeans(w, ng, length, mu, 40)
        piv, rk, it, _ = isdf.kmeans_select(isdf.Domain(length=length, num_grid=ng),
                                            torch.from_numpy(w).cuda(), mu, 40, rand_seed=1)
        assert (rk, it) == (rk_o, it_o)
        assert np.array_equal(piv, piv_o)


@pytest.mark.parametrize("ng,scale", [((24, 24, 24), 1.0), ((5, 7, 90), 1.0), ((31, 30, 2), 1.0),
                                      ((16, 15, 17), 1e-25), ((16, 15, 17), 1e22)])
def test_select_search_extremes_match_oracle(torch_cuda, ng, scale):
    """The shared candidate search where its portions, its single-precision
    distances and its seeds are at their limits: as many centroids as a few
    bricks hold, one, boxes thin and long, lengths whose squares leave single
    precision on either side, weights with dropped points."""
    torch = torch_cuda
    n = ng[0] * ng[1] * ng[2]
    length = tuple(scale * 0.37 * x for x in ng)
    w = np.random.default_rng(3).uniform(0.1, 1.0, n)
    w[n // 3:n // 3 + n // 7] = 0.0
    for mu in (1, 5, n // 3):
        piv_o, rk_o, it_o = port.kmeans(w, ng, length, mu, 12)
        piv, rk, it, _ = isdf.kmeans_select(isdf.Domain(length=length, num_grid=ng),
                                            torch.from_numpy(w).cuda(), mu, 12, rand_seed=1)
        assert (rk, it) == (rk_o, it_o)
        assert np.array_equal(piv, piv_o)


@pytest.mark.parametrize("mu", [2, 33, 700])
@pytest.mark.parametrize("ng", [(16, 16, 8), (40, 52, 1), (2051, 1, 1), (13, 17, 29)])
def test_select_empty_clusters_match_oracle(torch_cuda, ng, mu):
    """Empty-cluster compaction, counting-sort tiles with remainders and the
    nearest-point boxes: points with a few distinct places only (most weights
    dropped or the centroids' first points far from the rest), so that clusters
    empty at once; iteration caps of 0, 1, odd and even."""
    torch = torch_cuda
    n = ng[0] * ng[1] * ng[2]
    length = (4.0, 5.0, 6.0)
    rng = np.random.default_rng(n + mu)
    w = rng.uniform(0.5, 1.0, n) * np.exp(-rng.uniform(0.0, 17.0, n))
    w[mu // 2:mu] = 2.0 ** -30  # dropped or nearly so: centroids next to others
    for iters in (0, 1, 2, 7):
        piv_o, rk_o, it_o = port.kmeans(w, ng, length, mu, iters)
        piv, rk, it, _ = isdf.kmeans_select(isdf.Domain(length=length, num_grid=ng),
                                            torch.from_numpy(w).cuda(), mu, iters, rand_seed=1)
        assert (rk, it) == (rk_o, it_o)
        assert np.array_equal(piv, piv_o)


def test_select_ends_when_it_has_converged(torch_cuda):
    """Selections that converge within the first few iterations, under a cap far
    beyond them: no rounds of the loop behind the last iteration (the launches
    counted by the solve; for a batch, of which no count comes back, its time:
    a million rounds of idle launches take seconds)."""
    import time

    torch = torch_cuda
    g = load_golden("small_s1s2")
    psi, ng = g["psi"], tuple(int(x) for x in g["ng"])
    dom = isdf.Domain(length=tuple(float(x) for x in g["length"]), num_grid=ng)
    a = (int(g["nocc"]), psi.shape[1]) + tuple(int(g[k]) for k in ("nv1", "nc1", "nv2", "nc2"))
    d_psi = torch.from_numpy(np.ascontiguousarray(psi.T)).cuda()
    d_theta = torch.zeros((1, psi.shape[0]), dtype=torch.float64, device="cuda")
    few = None
    for cap in (20, 100000):
        piv = np.zeros(psi.shape[0], dtype=np.int32)
        torch.cuda.synchronize()
        rep = isdf.ISDF(d_psi, dom, *a, 1, d_theta, piv, cap)
        assert rep.rk_eff == 1 and rep.kmeans_iters <= 3
        few = few or rep.kernel_launches
        assert rep.kernel_launches <= few + 24  # a body of the loop or two more
    n = psi.shape[0]
    w = torch.zeros((3, n), dtype=torch.float64, device="cuda")
    w[:, 3:3 + 40 * 5:5] = 1.0  # as many kept points as centroids
    for mu in (40, 1):
        isdf.kmeans_select_batch([dom] * 3, list(w), [mu] * 3, [20] * 3, rand_seed=1)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        got = isdf.kmeans_select_batch([dom] * 3, list(w), [mu] * 3, [10 ** 6, 20, 10 ** 6],
                                       rand_seed=1)
        assert time.perf_counter() - t0 < 1.0
        assert all(it <= 3 for _, _, it, _ in got)


@pytest.mark.parametrize("cap", [2 ** 31 - 1, 2 ** 31 - 9])
def test_select_until_converged(torch_cuda, cap):
    """The largest iteration caps an int holds: 'until it converges', alone and as one
    request of a batch."""
    torch = torch_cuda
    ng, length = (13, 12, 11), (4.0, 5.0, 6.0)
    dom = isdf.Domain(length=length, num_grid=ng)
    w = np.random.default_rng(2).uniform(0.1, 1.0, ng[0] * ng[1] * ng[2])
    piv_o, rk_o, it_o = port.kmeans(w, ng, length, 37, 100000)
    assert it_o < 1000
    d_w = torch.from_numpy(w).cuda()
    piv, rk, it, _ = isdf.kmeans_select(dom, d_w, 37, cap, rand_seed=1)
    assert (rk, it) == (rk_o, it_o) and np.array_equal(piv, piv_o)
    got = isdf.kmeans_select_batch([dom] * 2, [d_w] * 2, [37] * 2, [3, cap], rand_seed=1)
    assert got[1][1:3] == (rk_o, it_o) and np.array_equal(got[1][0], piv_o)
    piv_o, rk_o, it_o = port.kmeans(w, ng, length, 37, 3)
    assert got[0][1:3] == (rk_o, it_o) and np.array_equal(got[0][0], piv_o)


def test_select_batch_groups_match_single(torch_cuda):
    """A batch of more than one launch's systems, of different grids, mu and
    iteration caps (one stops at once, one has fewer kept points than mu):
    every result equals the single selection's."""
    torch = torch_cuda
    rng = np.random.default_rng(11)
    doms, ws, mus, its = [], [], [], []
    for k in range(19):
        ng = tuple(int(x) for x in rng.integers(6, 25, 3))
        n = ng[0] * ng[1] * ng[2]
        w = rng.uniform(0.0, 1.0, n)
        w[rng.integers(0, n, n // 4)] = 0.0
        mu = int(rng.integers(1, min(513, n // 3)))
        if k == 7:
            w[:] = 0.0
            w[5:5 + mu // 2] = 1.0  # fewer kept points than mu
        doms.append(isdf.Domain(length=(5.0, 6.0, 7.0), num_grid=ng))
        ws.append(torch.from_numpy(w).cuda())
        mus.append(mu)
        its.append((0, 1, 30, 100)[k % 4])
    got = isdf.kmeans_select_batch(doms, ws, mus, its, rand_seed=1)
    for d, w, mu, it, g in zip(doms, ws, mus, its, got):
        one = isdf.kmeans_select(d, w, mu, it, rand_seed=1)
        assert g[1:] == one[1:]
        assert np.array_equal(g[0], one[0])


def test_loops_leave_the_callers_stream_to_others(torch_cuda):
    """Another thread launches on the stream that a selection runs on (alone, batched, by
    QRCP): what it launches runs once, and the selections stay what they are."""
    import threading

    torch = torch_cuda
    ng = (24, 23, 22)
    n = ng[0] * ng[1] * ng[2]
    dom = isdf.Domain(length=(5.0, 6.0, 7.0), num_grid=ng)
    w = np.random.default_rng(4).uniform(0.1, 1.0, n)
    d_w = torch.from_numpy(w).cuda()
    piv_o, rk_o, it_o = port.kmeans(w, ng, (5.0, 6.0, 7.0), 90, 40)
    psi = torch.from_numpy(np.random.default_rng(5).standard_normal((16, n))).cuda()
    theta = torch.empty((60, n), dtype=torch.float64, device="cuda")
    st = torch.cuda.Stream()
    opt = isdf.Options(stream=st.cuda_stream)
    piv_q = np.zeros(n, dtype=np.int32)
    torch.cuda.synchronize()
    isdf.ISDF(psi, dom, 8, 16, 8, 8, 8, 8, 60, theta, piv_q, 1, "QRCP", options=opt)
    added = torch.zeros(1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    stop, count, fail = threading.Event(), [0], []

    def others():
        try:
            with torch.cuda.stream(st):
                while not stop.wait(2e-5):
                    added.add_(1)
                    count[0] += 1
        except Exception as e:  # noqa: BLE001 - reported by the assertion below
            fail.append(repr(e))

    t = threading.Thread(target=others)
    t.start()
    try:
        for _ in range(30):
            piv, rk, it, _ = isdf.kmeans_select(dom, d_w, 90, 40, rand_seed=1,
                                                stream=st.cuda_stream)
            assert (rk, it) == (rk_o, it_o) and np.array_equal(piv, piv_o)
            got = isdf.kmeans_select_batch([dom] * 2, [d_w] * 2, [90] * 2, [40] * 2, rand_seed=1,
                                           stream=st.cuda_stream)
            assert all(g[1:3] == (rk_o, it_o) and np.array_equal(g[0], piv_o) for g in got)
            piv = np.zeros(n, dtype=np.int32)
            isdf.ISDF(psi, dom, 8, 16, 8, 8, 8, 8, 60, theta, piv, 1, "QRCP", options=opt)
            assert np.array_equal(piv, piv_q)
    finally:
        stop.set()
        t.join()
    torch.cuda.synchronize()
    assert not fail and count[0] > 0
    assert int(added) == count[0]


def test_loops_do_not_wait_for_other_streams(torch_cuda):
    """A selection (alone, batched, by QRCP) returns while a long copy to the host runs on
    another stream: a pipeline of solves overlaps the previous result's copy with the next
    solve. The copy takes tens of milliseconds, the calls a few."""
    torch = torch_cuda
    ng = (24, 23, 22)
    n = ng[0] * ng[1] * ng[2]
    dom = isdf.Domain(length=(5.0, 6.0, 7.0), num_grid=ng)
    d_w = torch.from_numpy(np.random.default_rng(4).uniform(0.1, 1.0, n)).cuda()
    psi = torch.from_numpy(np.random.default_rng(5).standard_normal((16, n))).cuda()
    theta = torch.empty((60, n), dtype=torch.float64, device="cuda")
    src = torch.zeros(3 << 30, dtype=torch.uint8, device="cuda")
    dst = torch.empty(3 << 30, dtype=torch.uint8, pin_memory=True)
    copies = torch.cuda.Stream()
    calls = {
        "single": lambda: isdf.kmeans_select(dom, d_w, 90, 40, rand_seed=1),
        "batch": lambda: isdf.kmeans_select_batch([dom] * 2, [d_w] * 2, [90] * 2, [40] * 2,
                                                  rand_seed=1),
        "qrcp": lambda: isdf.ISDF(psi, dom, 8, 16, 8, 8, 8, 8, 60, theta,
                                  np.zeros(n, dtype=np.int32), 1, "QRCP"),
    }
    for call in calls.values():
        call()  # the workspace, the kernels
    torch.cuda.synchronize()
    for name, call in calls.items():
        done = torch.cuda.Event()
        with torch.cuda.stream(copies):
            dst.copy_(src, non_blocking=True)
            done.record()
        call()
        running = not done.query()
        torch.cuda.synchronize()
        assert running, name


def test_select_ends_with_a_negative_tail(torch_cuda):
    """Weights are products of squares, but the caller's: a negative one at grid point 0,
    which the zero tail repeats in its cluster's sum, must not keep the sum from ending.
    One centroid, so that the sums decide nothing else."""
    torch = torch_cuda
    ng, length = (9, 8, 7), (4.0, 5.0, 6.0)
    n = ng[0] * ng[1] * ng[2]
    w = np.random.default_rng(1).uniform(0.1, 1.0, n)
    w[n // 2:] = 0.0
    w[0] = -2.0 ** -12
    piv_o, rk_o, it_o = port.kmeans(w, ng, length, 1, 10)
    piv, rk, it, _ = isdf.kmeans_select(isdf.Domain(length=length, num_grid=ng),
                                        torch.from_numpy(w).cuda(), 1, 10, rand_seed=1)
    assert (rk, it) == (rk_o, it_o)
    assert np.array_equal(piv, piv_o)

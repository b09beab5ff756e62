"""Fuzzy simplicial set, spectral initialisation and layout epochs on the GPU
against the reference's golden vectors and the CPU oracle."""

import numpy as np
import pytest
import torch

from oracle import fuzzy as ofz
from oracle import layout as olay
from oracle import spectral as ospec

pytestmark = pytest.mark.gpu


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def gpu_fuzzy(idx, dist, n_epochs, fp64):
    from mlx_vis_b200 import _lib

    r, c, v, ne, rho, sig = _lib.fuzzy(cuda(idx.astype(np.int32)), cuda(dist.astype(np.float32)), n_epochs,
                                       fp64=fp64, with_sigma=True)
    E = int(ne.item())
    return (r[:E].cpu().numpy(), c[:E].cpu().numpy(), v[:E].cpu().numpy()), (rho.cpu().numpy(), sig.cpu().numpy())


@pytest.mark.parametrize("name,n_epochs", [("fuzzy_gauss", 200), ("fuzzy_dups", 500)])
def test_fuzzy_fp64_matches_fp64_oracle(name, n_epochs, golden):
    g = golden(name)
    if name == "fuzzy_gauss":
        kb = golden("knn_brute_gauss")
        idx, dist = kb["idx"], kb["dist"]
    else:
        idx, dist = g["knn_idx"], g["knn_dist"]
    (r, c, v), (rho, sig) = gpu_fuzzy(idx, dist, n_epochs, fp64=True)
    (ro, co, vo), (rho_o, sig_o) = ofz.fuzzy_simplicial_set(idx, dist, n_epochs, dtype=np.float64)
    assert np.array_equal(r, ro) and np.array_equal(c, co)
    np.testing.assert_allclose(v, vo, rtol=1e-6)
    np.testing.assert_allclose(sig, sig_o.astype(np.float32), rtol=1e-6)
    # and against the reference (float32 bisection): same edge set, weights within its tolerance band
    assert np.array_equal(r, g["rows"]) and np.array_equal(c, g["cols"])
    rel = np.abs(v - g["vals"]) / g["vals"]
    assert rel.max() < 5e-5 and np.mean(rel < 1e-5) > 0.99


@pytest.mark.parametrize("name,n_epochs", [("fuzzy_gauss", 200), ("fuzzy_dups", 500)])
def test_fuzzy_fp32_mode_matches_reference(name, n_epochs, golden):
    g = golden(name)
    if name == "fuzzy_gauss":
        kb = golden("knn_brute_gauss")
        idx, dist = kb["idx"], kb["dist"]
    else:
        idx, dist = g["knn_idx"], g["knn_dist"]
    (r, c, v), _ = gpu_fuzzy(idx, dist, n_epochs, fp64=False)
    assert np.array_equal(r, g["rows"]) and np.array_equal(c, g["cols"])
    rel = np.abs(v - g["vals"]) / g["vals"]
    # expf and the row-sum order differ from NumPy's by ulps, which can move the
    # stopping point of a few rows inside the 1e-5 convergence band
    assert np.mean(rel <= 1e-5) > 0.99 and rel.max() < 5e-5


@pytest.fixture(params=["coop", "launches"])
def spectral_path(request, monkeypatch):
    """The power iteration runs as one cooperative launch unless UMAPB_SPECTRAL_COOP=0
    selects one launch per iteration; both must agree with the reference."""
    monkeypatch.setenv("UMAPB_SPECTRAL_COOP", "1" if request.param == "coop" else "0")
    return request.param


def test_spectral_matches_reference_with_injected_draws(golden, spectral_path):
    from mlx_vis_b200 import _lib

    fz, sp = golden("fuzzy_gauss"), golden("spectral_gauss")
    n = 2000
    rows, cols, vals = cuda(fz["rows"]), cuda(fz["cols"]), cuda(fz["vals"])
    ne = torch.tensor([rows.numel()], dtype=torch.int64, device="cuda")
    noise = np.random.RandomState(42).normal(scale=0.0001, size=(n, 2)).astype(np.float32)
    Y = _lib.spectral(rows, cols, vals, ne, n, 2, cuda(sp["V0"]), cuda(noise), n_iter=100,
                      check=True).cpu().numpy()
    Y64 = ospec.spectral_init(fz["rows"], fz["cols"], fz["vals"], n, sp["V0"], 0, dtype=np.float64)
    assert np.abs(Y - Y64).max() < 1e-4
    assert np.abs(Y - sp["Y0"]).max() < 1e-3


@pytest.mark.parametrize("dim", [1, 2, 3, 4])
def test_spectral_paths_agree_for_every_dim(golden, monkeypatch, dim):
    """Cooperative and per-iteration power iterations: same sums in FP64, the same
    embedding up to the order of the Gram matrix's atomic additions."""
    from mlx_vis_b200 import _lib

    fz = golden("fuzzy_gauss")
    n = 2000
    rows, cols, vals = cuda(fz["rows"]), cuda(fz["cols"]), cuda(fz["vals"])
    ne = torch.tensor([rows.numel()], dtype=torch.int64, device="cuda")
    V0 = np.random.RandomState(dim).normal(size=(n, dim + 1)).astype(np.float32)
    noise = np.random.RandomState(42).normal(scale=0.0001, size=(n, dim)).astype(np.float32)
    out = {}
    for path in ("1", "0"):
        monkeypatch.setenv("UMAPB_SPECTRAL_COOP", path)
        out[path] = _lib.spectral(rows, cols, vals, ne, n, dim, cuda(V0), cuda(noise), n_iter=100,
                                  check=True).cpu().numpy()
    assert out["1"].shape == (n, dim) and np.all(np.isfinite(out["1"]))
    assert np.abs(out["1"] - out["0"]).max() < 1e-3


@pytest.mark.parametrize("dim", [5, 8, 32])
def test_wide_spectral_matches_fp64_oracle(golden, dim):
    """n_components above 4: one launch per power iteration, one warp per row, the
    Gram matrix factored by the last block; against the FP64 oracle of umap.py:298-348."""
    from mlx_vis_b200 import _lib

    fz = golden("fuzzy_gauss")
    n = 2000
    rows, cols, vals = cuda(fz["rows"]), cuda(fz["cols"]), cuda(fz["vals"])
    ne = torch.tensor([rows.numel()], dtype=torch.int64, device="cuda")
    V0 = np.random.RandomState(dim).normal(size=(n, dim + 1)).astype(np.float32)
    noise = np.random.RandomState(42).normal(scale=0.0001, size=(n, dim)).astype(np.float32)
    Y = _lib.spectral(rows, cols, vals, ne, n, dim, cuda(V0), cuda(noise), n_iter=100, check=True).cpu().numpy()
    V = ospec.power_iteration(fz["rows"], fz["cols"], fz["vals"], n, V0, dtype=np.float64)
    Y64 = ospec.rescale(V[:, 1:].astype(np.float32), 42)
    assert Y.shape == (n, dim)
    # columns whose eigenvalues nearly coincide converge slowly in both; compare the
    # well-separated leading columns tightly and all columns on the whole
    assert np.abs(Y[:, :2] - Y64[:, :2]).max() < 1e-3
    assert np.median(np.abs(Y - Y64)) < 1e-3


def _layout(fz, n=2000, n_epochs=200, dim=2):
    from mlx_vis_b200 import _lib

    rows, cols, vals = cuda(fz["rows"]), cuda(fz["cols"]), cuda(fz["vals"])
    ne = torch.tensor([rows.numel()], dtype=torch.int64, device="cuda")
    return _lib.Layout(rows, cols, vals, ne, n, dim, n_epochs)


def test_schedule_active_counts_match_reference(golden, manifest):
    fz, opt = golden("fuzzy_gauss"), golden("optimize_gauss")
    m = manifest["optimize_gauss"]
    lay = _layout(fz)
    Y = cuda(opt["Y_ep0"].copy())
    counts = []
    for e in range(200):
        counts.append(lay.count_active(e))
        lay.epochs(Y, e, e + 1, m["a"], m["b"], 1.0, 5, 1234)
    assert counts == list(opt["n_active"])


def test_injected_epochs_match_reference(golden, manifest):
    fz, opt = golden("fuzzy_gauss"), golden("optimize_gauss")
    m = manifest["optimize_gauss"]
    lay = _layout(fz)
    Y = cuda(opt["Y_ep0"].copy())
    nonempty = [e for e in range(200) if opt["n_active"][e] > 0]
    assert nonempty[:2] == [1, 2]  # the fixture holds snapshots after epochs 1 and 2 (Y_ep2, Y_ep3)
    scale = float(np.abs(opt["Y_ep0"]).max())
    for j, e in enumerate(nonempty[:2]):
        # epochs before the first non-empty one do nothing
        lay.epochs(Y, (nonempty[j - 1] + 1) if j else 0, e, m["a"], m["b"], 1.0, 5, 0)
        lay.epoch_injected(Y, e, m["a"], m["b"], 1.0, 5, cuda(opt[f"neg_{j}"].astype(np.int32)))
        if j == 0:
            got = Y.cpu().numpy()
            ref = opt[f"Y_ep{e + 1}"]
            # one epoch: within 1e-5 of the reference coordinates (relative to their scale)
            assert np.abs(got - ref).max() <= 1e-5 * max(1.0, scale), np.abs(got - ref).max()
            sets = olay.active_sets(fz["vals"], 200)
            Yo = olay.sgd_epoch(opt["Y_ep0"], fz["rows"][sets[e]], fz["cols"][sets[e]],
                                np.resize(fz["rows"][sets[e]], 5 * len(sets[e])), opt["neg_0"].astype(np.int64),
                                1.0 * (1 - e / 200), m["a"], m["b"])
            assert np.abs(got - Yo).max() <= 1e-5 * max(1.0, scale)
    got = Y.cpu().numpy()
    ref = opt["Y_ep3"]
    # after a second epoch the steep short-range forces amplify rounding; stay close
    assert np.median(np.abs(got - ref)) < 1e-5 and np.abs(got - ref).max() < 1e-2


@pytest.mark.parametrize("dim", [5, 8, 32])
def test_wide_injected_epoch_matches_oracle(golden, manifest, dim):
    """One epoch at n_components above 4 (one warp per edge) with injected tails,
    against the FP32 oracle of umap.py:359-387."""
    fz, opt = golden("fuzzy_gauss"), golden("optimize_gauss")
    m = manifest["optimize_gauss"]
    lay = _layout(fz, dim=dim)
    rng = np.random.default_rng(dim)
    Y0 = rng.uniform(0, 10, size=(2000, dim)).astype(np.float32)
    Y = cuda(Y0.copy())
    sets = olay.active_sets(fz["vals"], 200)
    e = next(t for t in range(200) if len(sets[t]) > 0)
    lay.epochs(Y, 0, e, m["a"], m["b"], 1.0, 5, 0)
    A = len(sets[e])
    neg = rng.integers(0, 2000, 5 * A).astype(np.int32)
    lay.epoch_injected(Y, e, m["a"], m["b"], 1.0, 5, cuda(neg))
    got = Y.cpu().numpy()
    Yo = olay.sgd_epoch(Y0, fz["rows"][sets[e]], fz["cols"][sets[e]], np.resize(fz["rows"][sets[e]], 5 * A),
                        neg.astype(np.int64), 1.0 * (1 - e / 200), m["a"], m["b"])
    assert np.abs(got - Y0).max() > 1e-3  # the epoch moved the points
    assert np.abs(got - Yo).max() <= 1e-4, np.abs(got - Yo).max()


def test_injected_negative_count_is_checked(golden, manifest):
    from mlx_vis_b200 import _lib

    fz, opt = golden("fuzzy_gauss"), golden("optimize_gauss")
    m = manifest["optimize_gauss"]
    lay = _layout(fz)
    Y = cuda(opt["Y_ep0"].copy())
    with pytest.raises(_lib.UmapB200Error, match="negatives are needed"):
        lay.epoch_injected(Y, 1, m["a"], m["b"], 1.0, 5, cuda(opt["neg_0"][:-5].astype(np.int32)))


@pytest.mark.parametrize("parallel", [True, False])
@pytest.mark.parametrize("seed,shape", [(42, (70000, 2)), (0, (1, 3)), (7, (2001, 2)), (3, (1, 1))])
def test_device_legacy_normal_equals_numpy(seed, shape, parallel):
    """The spectral init's noise, RandomState(seed).normal(scale=1e-4) as float32,
    drawn on the device from the stream's state, bit for bit."""
    from mlx_vis_b200 import _lib

    want = np.random.RandomState(seed).normal(scale=0.0001, size=shape).astype(np.float32)
    got = _lib.legacy_normal(np.random.RandomState(seed), shape, 0.0, 0.0001, torch.device("cuda"), parallel=parallel)
    assert np.array_equal(got.cpu().numpy(), want)


def test_graph_epochs_match_launched_epochs(golden, manifest, monkeypatch):
    """umapb_layout_epochs_graph (recorded once, then updated in place for a new
    layout, and for another rate and seed) reaches the same coordinates as the
    launch-by-launch loop; float atomics may add the moves of one point in another order, hence the
    tolerance.  So few rows would otherwise be one launch, which records no graph."""
    monkeypatch.setenv("UMAPB_LAYOUT_ONE_LAUNCH", "0")
    fz, opt = golden("fuzzy_gauss"), golden("optimize_gauss")
    m = manifest["optimize_gauss"]
    for rate, seed in ((1.0, 7), (0.5, 8)):
        outs = []
        for graph in (False, True, True):  # the second graph call updates the cached executable
            lay = _layout(fz)
            Y = cuda(opt["Y_ep0"].copy())
            lay.epochs(Y, 0, 6, m["a"], m["b"], rate, 5, seed, graph=graph)
            outs.append(Y.cpu().numpy())
        scale = float(np.abs(outs[0]).max())
        assert np.abs(outs[0] - opt["Y_ep0"]).max() > 1e-3 * scale  # the epochs moved the points
        for o in outs[1:]:
            assert np.median(np.abs(o - outs[0])) < 1e-5 * scale
            assert np.abs(o - outs[0]).max() < 1e-2 * scale


@pytest.mark.parametrize("form", ["", "0"])
@pytest.mark.parametrize("dim", [2, 3])
def test_neg5_kernel_matches_general_kernel(golden, manifest, monkeypatch, dim, form):
    """At the default 5 negatives per edge the epochs run on a kernel compiled for that
    rate (UMAPB_LAYOUT_NEG5=0 selects the general kernel), in one launch and by launches:
    both draw the same tails and make the same sums, so only the order of the float atomics
    may differ."""
    monkeypatch.setenv("UMAPB_LAYOUT_ONE_LAUNCH", form)
    fz, opt = golden("fuzzy_gauss"), golden("optimize_gauss")
    m = manifest["optimize_gauss"]
    Y0 = opt["Y_ep0"]
    if dim != Y0.shape[1]:
        Y0 = np.concatenate([Y0, Y0[:, :1] * 0.5], axis=1)[:, :dim].astype(np.float32)
    outs = []
    for flag in ("1", "0"):
        monkeypatch.setenv("UMAPB_LAYOUT_NEG5", flag)
        lay = _layout(fz, dim=dim)
        Y = cuda(Y0.copy())
        lay.epochs(Y, 0, 6, m["a"], m["b"], 1.0, 5, 11, graph=False)
        outs.append(Y.cpu().numpy())
    scale = float(np.abs(outs[0]).max())
    assert np.abs(outs[0] - Y0).max() > 1e-3 * scale
    assert np.median(np.abs(outs[1] - outs[0])) < 1e-5 * scale
    assert np.abs(outs[1] - outs[0]).max() < 1e-2 * scale


@pytest.mark.parametrize("n,k,dim", [(17, 16, 2), (300, 5, 1), (300, 40, 4), (2560, 12, 4), (2561, 12, 4),
                                     (5120, 9, 2), (5121, 9, 2), (9000, 24, 3), (6000, 140, 2), (2048, 40, 2), (2048, 60, 4),
                                     (2049, 9, 4), (2049, 60, 3), (4096, 16, 3), (4097, 16, 2), (2000, 100, 2),
                                     (2000, 200, 2), (33, 300, 2), (60000, 130, 1)])
def test_power_iteration_forms_match_float64(n, k, dim):
    """The cluster form (one pass of 2,048 rows whose edges fit shared memory; up to 4,096 rows of
    16 bytes with 40,000 edges) and the grid-wide one (blocks by rows, by edges and by
    warps) on either side of their borders, uneven row counts per CTA and more edges than a CTA's
    shared memory was sized for, against float64 torch.  FP32 storage of V leaves 100
    rounded steps: 1e-5 of the 0..10 range."""
    from mlx_vis_b200 import _lib

    rng = np.random.default_rng(n + dim)
    deg = np.where(np.arange(n) < n // 4, k, np.maximum(1, k // 4))  # the first quarter has most of the edges
    rows = np.repeat(np.arange(n), deg).astype(np.int32)
    near = (rows + rng.integers(1, min(n - 1, 40) + 1, size=rows.size)) % n
    cols = near.astype(np.int32)
    vals = rng.uniform(0.2, 1.0, size=rows.size).astype(np.float32)
    V0 = rng.normal(size=(n, dim + 1)).astype(np.float32)
    noise = (1e-4 * rng.normal(size=(n, dim))).astype(np.float32)
    ne = torch.tensor([rows.size], dtype=torch.int64, device="cuda")
    Y = _lib.spectral(cuda(rows), cuda(cols), cuda(vals), ne, n, dim, cuda(V0), cuda(noise), n_iter=100,
                      check=True).cpu().numpy()
    r, c, w = torch.from_numpy(rows).long(), torch.from_numpy(cols).long(), torch.from_numpy(vals).double()
    d = torch.zeros(n, dtype=torch.float64).index_add_(0, r, w).clamp_min(1e-10)
    wn = w / (d[r] * d[c]).sqrt()
    V = torch.from_numpy(V0).double()
    for _ in range(100):
        V = torch.zeros_like(V).index_add_(0, r, wn[:, None] * V[c])
        V, R = torch.linalg.qr(V)
        V = V * R.diagonal().sign()  # the reference's norms are positive
    e = V[:, 1:]
    e = e * (10.0 / e.abs().max()) + torch.from_numpy(noise).double()
    want = (10.0 * (e - e.amin(0)) / (e.amax(0) - e.amin(0) + 1e-10)).numpy()
    assert np.abs(Y - want).max() < 1e-4


@pytest.mark.parametrize("n,k", [(40, 2), (333, 9), (333, 10), (1000, 66), (40000, 17), (40000, 18), (1000, 4),
                                 (40001, 9), (40001, 10), (16384, 16), (16385, 18), (20001, 20), (20001, 34), (20001, 40),
                                 (40001, 41), (40001, 64)])
def test_fuzzy_lanes_match_float64(n, k):
    """The bisection with 1, 2, 4 and 8 lanes per row, by rows and neighbours: neighbours on either
    side of the gaps a lane keeps in registers, rows with equal and with zero distances."""
    rng = np.random.default_rng(n + k)
    dist = np.sort(rng.uniform(0.5, 3.0, size=(n, k)), axis=1).astype(np.float32)
    dist[::7, : k // 2] = 0.0
    dist[::11] = 1.25
    idx = ((np.arange(n)[:, None] + 1 + np.arange(k)) % n).astype(np.int32)
    (r, c, v), _ = gpu_fuzzy(idx, dist, 200, fp64=True)
    (ro, co, vo), _ = ofz.fuzzy_simplicial_set(idx, dist, 200, dtype=np.float64)
    assert np.array_equal(r, ro) and np.array_equal(c, co)
    np.testing.assert_allclose(v, vo, rtol=1e-6)


@pytest.mark.parametrize("n,k,dim,neg", [(2, 1, 2, 5), (17, 3, 1, 5), (513, 7, 2, 5), (700, 9, 3, 5), (300, 5, 4, 2),
                                         (2000, 15, 2, 0), (1025, 11, 2, 11), (1228, 10, 2, 5), (1229, 10, 2, 5), (4000, 9, 1, 5),
                                         (20, 1600, 2, 5), (3000, 20, 4, 3), (20000, 15, 2, 5), (13001, 15, 3, 5),
                                         (30001, 5, 2, 5), (18501, 21, 3, 10), (56001, 3, 1, 0), (70003, 15, 2, 5), (70003, 24, 2, 5), (80003, 15, 3, 5), (70003, 15, 2, 3)])
@pytest.mark.parametrize("graph", [False, True])
def test_layout_many_epochs_match_single_epochs(n, k, dim, neg, graph):
    """Epochs 3 to 12 in one call (one launch up to 12,288 edges on a cluster, beyond on a resident
    grid; from about 55,000 values of Y on, launches that overlap) against the same epochs one
    call each (launches that do not): the same due edges and draws; a small step keeps the sums'
    order from growing.  Either side of each border, every narrow dimension, no and many
    negatives, one and several passes of a warp, uneven last shares; the schedule goes on after it."""
    from mlx_vis_b200 import _lib

    rng = np.random.default_rng(n + k)
    E = n * k - n * k // 7  # fewer edges than the arrays have room for
    rows = np.sort(rng.integers(0, n, size=n * k)).astype(np.int32)
    cols = rng.integers(0, n, size=n * k).astype(np.int32)
    vals = rng.uniform(0.05, 1.0, size=n * k).astype(np.float32)
    ne = torch.tensor([E], dtype=torch.int64, device="cuda")
    Y0 = cuda((10 * rng.normal(size=(n, dim))).astype(np.float32))
    # an epoch pulls a row by up to 2ab = 2.8 rate per edge that lists it, 2 k of them: above 1 in
    # all, a difference of the last bit grows from epoch to epoch instead of dying out
    rate = min(0.01, 0.5 / (2.8 * 2 * k))
    out = []
    for calls in ([(3, 12), (12, 13)], [(e, e + 1) for e in range(3, 13)]):
        lay = _lib.Layout(cuda(rows), cuda(cols), cuda(vals), ne, n, dim, 200)
        Y = Y0.clone()
        for b, e in calls:
            lay.epochs(Y, b, e, 1.577, 0.895, rate, neg, 12345, graph=graph)
        out.append((Y.cpu().numpy(), lay.next[:E].cpu().numpy()))
    assert np.array_equal(out[0][1], out[1][1])
    # float32 sums of up to (1 + neg) k clipped moves of at most 0.04 per epoch, in another order
    scale = np.abs(Y0.cpu().numpy()).max()
    assert np.abs(out[0][0] - out[1][0]).max() < 2e-5 * scale


@pytest.mark.parametrize("graph", [False, True])
def test_layout_barrier_that_gives_up_changes_nothing(graph):
    """The resident grid's barrier with a limit of 1 ns: the launch ends with the status word set, Y
    and the schedule as they were, and the same epochs run by launches from there."""
    from mlx_vis_b200 import _lib

    n, k = 4000, 9  # 36,000 edges: a grid, not a cluster
    rng = np.random.default_rng(5)
    rows = np.sort(rng.integers(0, n, size=n * k)).astype(np.int32)
    cols = rng.integers(0, n, size=n * k).astype(np.int32)
    vals = rng.uniform(0.05, 1.0, size=n * k).astype(np.float32)
    ne = torch.tensor([n * k], dtype=torch.int64, device="cuda")
    Y0 = cuda((10 * rng.normal(size=(n, 2))).astype(np.float32))
    args = (1.577, 0.895, 0.01, 5, 12345)
    lay, want = (_lib.Layout(cuda(rows), cuda(cols), cuda(vals), ne, n, 2, 200) for _ in range(2))
    Y, Yw, next0 = Y0.clone(), Y0.clone(), lay.next.clone()
    try:
        _lib.set_wait_limit_ns(1)
        lay.epochs(Y, 0, 12, *args, graph=graph)
        torch.cuda.synchronize()
    finally:
        _lib.set_wait_limit_ns(0)
    assert _lib.status_word(lay.ws) == 3
    assert torch.equal(Y, Y0) and torch.equal(lay.next, next0)
    with pytest.raises(_lib.UmapB200Error):
        lay.check()
    lay.check()  # told once
    lay.epochs_by_launches(Y, 0, 12, *args)
    want.epochs(Yw, 0, 12, *args)  # one launch
    want.check()
    assert torch.equal(lay.next, want.next)
    assert float((Yw - Y0).abs().max()) > 1e-3
    assert float((Y - Yw).abs().max()) < 2e-5 * float(Y0.abs().max())  # float32 sums in another order


def test_fit_goes_on_by_launches_when_the_layout_gives_up(gauss2000):
    """fit_transform with a layout whose barrier expires: the same embedding by launches.  Even at a
    limit of 1 ns every CTA of a fit can find the others there, so some fits may be needed."""
    from mlx_vis_b200 import UMAP, _lib

    def fit(limit):
        try:
            _lib.set_wait_limit_ns(limit)
            before = _lib.kernel_launches()
            # a random start: the spectral one has a barrier with the same limit
            Y = UMAP(n_epochs=20, learning_rate=0.05, init="random", knn_method="brute",
                     random_state=4).fit_transform(gauss2000)
            return Y, _lib.kernel_launches() - before
        finally:
            _lib.set_wait_limit_ns(0)

    want, launches = fit(0)
    for _ in range(40):
        Y, took = fit(1)
        assert np.linalg.norm(Y - want) < 1e-3 * np.linalg.norm(want)  # sums in another order over 20 epochs
        if took != launches:
            break
    assert took == launches + 40  # two launches an epoch besides the one that gave up


@pytest.mark.parametrize("form", ["", "grid", "0"])
def test_layout_without_edges(monkeypatch, form):
    """No edge and no room for one, in every form of the epochs: Y stays."""
    from mlx_vis_b200 import _lib

    monkeypatch.setenv("UMAPB_LAYOUT_ONE_LAUNCH", form)
    one = torch.zeros(1, dtype=torch.int32, device="cuda")
    ne = torch.zeros(1, dtype=torch.int64, device="cuda")
    lay = _lib.Layout(one, one, torch.zeros(1, device="cuda"), ne, 50, 2, 20)
    lay.e_cap = 0
    Y0 = cuda(np.random.default_rng(0).normal(size=(50, 2)).astype(np.float32))
    Y = Y0.clone()
    lay.epochs(Y, 0, 6, 1.577, 0.895, 1.0, 5, 3)
    lay.check()
    assert torch.equal(Y, Y0)


def test_fuzzy_drops_missing_neighbours():
    """Where scores overflow, the exact search fills a row with the id 0x7fffffff at an infinite distance:
    no edge points there, and the others keep their weights."""
    n, k = 300, 6
    rng = np.random.default_rng(1)
    idx = ((np.arange(n)[:, None] + 1 + np.arange(k)) % n).astype(np.int32)
    dist = np.sort(rng.uniform(0.5, 3.0, size=(n, k)), axis=1).astype(np.float32)
    idx[:20], dist[:20] = 0x7FFFFFFF, np.inf  # rows without any neighbour
    idx[20:40, -1], dist[20:40, -1] = 0x7FFFFFFF, np.inf  # and with one less
    idx[40, -1] = -1
    (r, c, v), _ = gpu_fuzzy(idx, dist, 200, fp64=True)
    assert c.min() >= 0 and c.max() < n and r.min() >= 20 and not np.isnan(v).any()
    whole = ((np.arange(n)[:, None] + 1 + np.arange(k)) % n).astype(np.int32)
    (ro, co, vo), _ = ofz.fuzzy_simplicial_set(whole, np.where(np.isinf(dist), np.float32(1e6), dist), 200,
                                               dtype=np.float64)
    # rows at a distance from the altered ones, whose neighbours are as they were
    a, b = (r >= 60) & (r < n - 10), (ro >= 60) & (ro < n - 10)
    assert np.array_equal(r[a], ro[b]) and np.array_equal(c[a], co[b])
    np.testing.assert_allclose(v[a], vo[b], rtol=1e-6)


def test_fit_of_rows_that_overflow():
    """Squared norms beyond FP32 leave rows without neighbours: the fit ends with every other row embedded."""
    from mlx_vis_b200 import UMAP

    X = np.random.default_rng(0).normal(size=(400, 12)).astype(np.float32)
    X[::40] *= 1e25
    Y = UMAP(n_epochs=20, knn_method="brute", random_state=0).fit_transform(X)
    assert Y.shape == (400, 2)

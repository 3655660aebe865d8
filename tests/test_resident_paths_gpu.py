"""The step paths that keep a network resident (cluster, grid, adjoint grid
segments) and the launches around them, at the sizes where their splits change:
edges of tiles, CTAs and launch rules, ragged and edgeless networks, zero
delays, blocks longer than one launch (GPU).

Forward results, hub counts and weight conversions are compared with the
per-step kernels bit for bit.  Gradients are compared at a relative difference
of 1e-5: between paths only the order of the sums over edges and of the
float32 scatters differs (some tens of terms of one sign pattern each, so a few
1e-7 per sum; dL/dK, a sum over nodes and steps that cancels, has differed by
5.7e-6 in 60,000 pairs of runs).
"""

import numpy as np
import pytest
import torch

from adjoint64 import simulate as simulate64
from conftest import has_gpu
from leviathan_v1_b200 import BatchEngine, HubTransitions, LeviathanEngine, _lib
from leviathan_v1_b200.adjoint import Adjoint, simulate
from leviathan_v1_b200.graphs import Network, init_state, make_network

pytestmark = pytest.mark.gpu

DT = 0.05
REL = 1e-5


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not has_gpu():
        pytest.fail("GPU tests need a CUDA device")


def _state(e):
    th_hat, om_hat = e.get_predictor()
    out = dict(theta=e.get_all_theta(), w=e.get_weights(), thh=th_hat, omh=om_hat)
    for k in range(e.num_nets):
        ring, bi = e.get_ring(k)
        out[f"ring{k}"], out[f"bi{k}"] = ring, np.array(bi)
        out[f"g{k}"] = np.array(e._get_gain(k))
        out[f"t{k}"] = np.array(e.step_count(k))
    return out


def _same(a, b, what=""):
    for k, v in b.items():
        np.testing.assert_array_equal(a[k], v, err_msg=f"{what}{k}")


def _per_step(e):
    e.set_cluster_mode(False)
    e.set_grid_mode(False)
    e.set_pair_mode(False)
    return e


def _from_degrees(deg, max_delay, seed):
    """Directed network with the given in-degrees, sources drawn at random."""
    rng = np.random.default_rng(seed)
    n = len(deg)
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    col = np.concatenate([np.sort(rng.choice(n, d, replace=False)) for d in deg]
                         + [np.zeros(0, int)]).astype(np.int32)
    st = init_state(rp, max_delay, seed)
    return Network(n, max_delay, rp, col, st["delays"], st["weights"], st["theta"],
                   st["theta_hat"], st["omega"])


def _uneven(seed, zero):
    """Networks of 1 to 2,049 rows: one row, a part of a warp, a tile and one
    row, without edges, with rows of 0 to 90 entries, and one zero delay or
    none."""
    rng = np.random.default_rng(seed)
    lo = 0 if zero else 1
    return [_from_degrees(np.zeros(1, int), 3, seed),
            make_network(33, 4, 0.1, 6, seed=seed + 1, delay_lo=1),
            make_network(257, 8, 0.1, 20, seed=seed + 2, delay_lo=1),
            _from_degrees(np.zeros(300, int), 5, seed + 3),
            _from_degrees(np.where(np.arange(700) % 97 == 0, 90, rng.integers(0, 12, 700)),
                          17, seed + 4),
            make_network(2049, 16, 0.1, 9, seed=seed + 5, delay_lo=lo)]


@pytest.mark.parametrize("mode,zero", [("reference", False), ("accurate", False),
                                       ("reference", True)])
def test_batch_on_the_grid_kernel(mode, zero):
    nets = [n.as_dict() for n in _uneven(5, zero)]
    params = [dict(g=0.3 * (i + 1), gain_controller=i % 2) for i in range(len(nets))]
    ref = _per_step(BatchEngine(nets, params=params, math_mode=mode))
    want_r = np.concatenate([ref.step_n(DT, 5), ref.step_n(DT, 70)])
    want = _state(ref)
    ref.close()
    e = BatchEngine(nets, params=params, math_mode=mode)
    rows = e.grid_info()["eligible_rows"]
    e.close()
    assert rows
    for R in rows:
        e = BatchEngine(nets, params=params, math_mode=mode)
        e.set_grid_mode(True, R)
        assert e.grid_info()["enabled"]
        r = np.concatenate([e.step_n(DT, 5), e.step_n(DT, 70)])
        np.testing.assert_array_equal(r, want_r, err_msg=f"R={R}")
        _same(_state(e), want, f"R={R}: ")
        e.close()


# one CTA; two CTAs per SM exactly (148 SMs) and one CTA more, where the exchange
# goes from two warps to one
@pytest.mark.parametrize("N,k,R", [(33, 4, 64), (129, 30, 128), (18_944, 8, 64), (18_945, 8, 64),
                                   (37_888, 4, 128), (37_889, 4, 128)])
def test_grid_kernel_at_the_edges_of_its_split(N, k, R):
    net = make_network(N, k, 0.1, 11, seed=N, delay_lo=1)
    ref = _per_step(LeviathanEngine(*net.engine_args()))
    want_r = ref.step_n(DT, 40)
    want = _state(ref)
    ref.close()
    e = LeviathanEngine(*net.engine_args())
    if R not in e.grid_info()["eligible_rows"]:
        e.close()
        pytest.skip("these rows per CTA do not fit this device")
    e.set_cluster_mode(False)
    e.set_grid_mode(True, R)
    np.testing.assert_array_equal(e.step_n(DT, 40), want_r)
    _same(_state(e), want)
    e.close()


@pytest.mark.parametrize("N,R,lo", [(1000, 0, 1), (1000, 0, 0), (5000, 64, 1), (5000, 256, 1),
                                    (5000, 64, 0), (5000, 256, 0)])
def test_hubs_on_resident_paths(N, R, lo):
    """R = 0: the cluster kernel."""
    net = make_network(N, 12, 0.1, 20, seed=N + R + lo, delay_lo=lo)
    hubs = [0, N - 1, 31, 32, 255, 256, N // 2]
    out = []
    for resident in (False, True):
        e = LeviathanEngine(*net.engine_args())
        m = HubTransitions(hubs)
        m.attach(e)
        if resident:
            e.set_cluster_mode(R == 0)
            e.set_grid_mode(R > 0, R)
            assert R == 0 or e.grid_info()["enabled"]
        else:
            _per_step(e)
        r = np.concatenate([e.step_n(DT, 37), [e.step(DT)], e.step_n(DT, 1), e.step_n(DT, 90)])
        out.append((r, *m.read(), e.get_theta()))
        m.close()
        e.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    assert out[1][4] == 129  # every step observed


def test_hubs_of_one_network_of_a_resident_batch():
    nets = [n.as_dict() for n in _uneven(9, False)]
    out = []
    for resident in (False, True):
        e = BatchEngine(nets)
        m = HubTransitions([0, 699, 255, 256])
        m.attach(e, net=4)
        if resident:
            e.set_grid_mode(True)
            assert e.grid_info()["enabled"]
        else:
            _per_step(e)
        out.append((e.step_n(DT, 60), *m.read()))
        m.close()
        e.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("lo", [1, 0])
def test_cluster_wait_timeout_is_reported(lo):
    """A wait that runs out (20 us, one arrival more than ever comes) ends the
    launch with an error; the engine goes on with per-step launches from the
    state before."""
    net = make_network(1000, 20, 0.1, 30, seed=3, delay_lo=lo)
    ref = _per_step(LeviathanEngine(*net.engine_args()))
    want_r = np.concatenate([ref.step_n(DT, 7), ref.step_n(DT, 40)])
    want = _state(ref)
    ref.close()
    e = LeviathanEngine(*net.engine_args())
    e.set_cluster_mode(True)
    np.testing.assert_array_equal(e.step_n(DT, 7), want_r[:7])
    e.set_grid_wait(20_000, extra_arrivals=1)
    with pytest.raises(_lib.LevError) as exc:
        e.step_n(DT, 40)
    assert exc.value.code == _lib.LEV_ERR_CUDA and "timed out" in str(exc.value)
    e.set_grid_wait()
    np.testing.assert_array_equal(e.step_n(DT, 40), want_r[7:])
    _same(_state(e), want)
    e.close()


@pytest.mark.parametrize("N,k,cluster", [(300, 8, True), (3000, 8, False)])
def test_blocks_longer_than_one_resident_launch(N, k, cluster):
    """2,100 steps: more than the 2,048 one launch takes."""
    net = make_network(N, k, 0.1, 12, seed=N, delay_lo=1)
    ref = LeviathanEngine(*net.engine_args())
    ref.set_cluster_mode(False)
    ref.set_grid_mode(False)
    want_r = ref.step_n(DT, 2100)
    want = _state(ref)
    ref.close()
    e = LeviathanEngine(*net.engine_args())
    e.set_cluster_mode(cluster)
    e.set_grid_mode(not cluster)
    np.testing.assert_array_equal(e.step_n(DT, 2100), want_r)
    _same(_state(e), want)
    e.close()


def test_engines_of_different_sizes_share_the_kernels():
    """A smaller engine made later leaves the larger one's launches valid."""
    nets = [make_network(16_000, 20, 0.1, 30, seed=1, delay_lo=1),
            make_network(1000, 20, 0.1, 30, seed=2, delay_lo=1),
            make_network(200, 4, 0.1, 5, seed=3, delay_lo=1)]
    for cluster in (False, True):
        es = [LeviathanEngine(*n.engine_args()) for n in nets]
        for e, n in zip(es, nets):
            if cluster and not e.cluster_info()["eligible"]:
                continue
            e.set_cluster_mode(cluster)
            ref = _per_step(LeviathanEngine(*n.engine_args()))
            np.testing.assert_array_equal(e.step_n(DT, 20), ref.step_n(DT, 20))
            ref.close()
        for e in es:
            e.close()


# tiles of 256 rows at the limits of the dependent launches: one, 111 | 112,
# 444 | 445
@pytest.mark.parametrize("N", [200, 28_416, 28_417, 113_664, 113_665])
def test_pair_chain_at_the_limits_of_its_launch_rule(N):
    net = make_network(N, 4, 0.1, 7, seed=N, delay_lo=1)
    ref = _per_step(LeviathanEngine(*net.engine_args()))
    want_r = ref.step_n(DT, 21)
    want = _state(ref)
    ref.close()
    e = LeviathanEngine(*net.engine_args())
    e.set_cluster_mode(False)
    e.set_grid_mode(False)
    assert any(c["enabled"] for c in e.pair_info())
    np.testing.assert_array_equal(e.step_n(DT, 21), want_r)
    _same(_state(e), want)
    e.close()


@pytest.mark.parametrize("batch", [False, True])
def test_weights_round_trip(batch):
    nets = _uneven(13, True) if batch else _uneven(13, True)[4:5]
    e = BatchEngine([n.as_dict() for n in nets])
    np.testing.assert_array_equal(e.get_weights(), np.concatenate([n.weights for n in nets]))
    w = np.random.default_rng(0).random(sum(len(n.weights) for n in nets)).astype(np.float32)
    e.reset_weights(w)
    np.testing.assert_array_equal(e.get_weights(), w)
    e.close()


def _rel(a, b):
    a, b = a.double().cpu().numpy().ravel(), b.double().cpu().numpy().ravel()
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)


# one segment; a last segment of one step; several and a part; 2,200 rows take the
# split step kernels, 40,000 (over 148 tiles) the one-lane ones
@pytest.mark.parametrize("N,T,segment", [(2200, 30, 50), (2200, 51, 25), (2200, 60, 25),
                                         (40_000, 21, 10), (40_000, 24, 10)])
def test_gradients_from_the_recorded_last_segment(N, T, segment):
    """The forward pass keeps its last segment's records; a second backward
    pass, and one on another path than the forward pass, recompute them."""
    net = make_network(N, 8, 0.1, 9, seed=N + T, delay_lo=1)
    om, w0 = (torch.tensor(x, device="cuda") for x in (net.omega, net.weights))
    K = torch.full((1,), 1.5, device="cuda")
    dr = torch.linspace(-1, 1, T, device="cuda")[:, None].contiguous()

    def run(forward_grid, backward_grid, twice=False):
        eng = LeviathanEngine(*net.engine_args())
        adj = Adjoint(eng, segment=segment, max_steps=T)
        adj.set_grid_mode(forward_grid)
        r = adj.forward(om, w0, K, T, DT)
        adj.set_grid_mode(backward_grid)
        out = [adj.backward(dr)]
        if twice:
            out.append(adj.backward(dr))
        adj.close()
        eng.close()
        return r, out

    r_ref, (_, ref) = run(False, False, twice=True)  # recomputed throughout
    for f, b in [(False, False), (True, True), (True, False), (False, True)]:
        r, out = run(f, b, twice=f and b)
        assert torch.equal(r, r_ref)
        for g in out:
            for k in ("omega", "w0", "K"):
                assert _rel(g[k], ref[k]) <= REL, (f, b, k)


# 18,945 rows: one CTA of 64 rows more than two per SM
@pytest.mark.parametrize("N,k,lo,mode", [(65, 4, 1, "reference"), (2049, 30, 0, "reference"),
                                         (2049, 30, 1, "accurate"), (18_945, 4, 1, "reference")])
def test_adjoint_grid_segments_at_ragged_sizes(N, k, lo, mode):
    net = make_network(N, k, 0.1, 6, seed=N + lo, delay_lo=lo)
    om, w0 = (torch.tensor(x, device="cuda") for x in (net.omega, net.weights))
    K = torch.full((1,), 1.5, device="cuda")
    T = 27
    dr = torch.linspace(-1, 1, T, device="cuda")[:, None].contiguous()
    eng = LeviathanEngine(*net.engine_args(), math_mode=mode)
    adj = Adjoint(eng, segment=10, max_steps=T)
    rows = adj.grid_info()["eligible_rows"]
    assert rows
    adj.set_grid_mode(False)
    r_ref, ref = adj.forward(om, w0, K, T, DT), adj.backward(dr)
    for R in rows:
        for paired in (False, True):
            adj.set_grid_mode(True, R)
            adj.set_grid_pairing(paired)
            assert torch.equal(adj.forward(om, w0, K, T, DT), r_ref)
            g = adj.backward(dr)
            for name in ("omega", "w0", "K"):
                assert _rel(g[name], ref[name]) <= REL, (R, paired, name)
    adj.close()
    eng.close()


@pytest.mark.parametrize("k,mode", [(5, "reference"), (9, "reference"), (9, "accurate"),
                                    (12, "reference"), (13, "reference"), (24, "reference"),
                                    (25, "accurate"), (25, "reference"), (36, "reference"),
                                    (37, "reference")])
def test_one_lane_per_row_at_the_edges_of_its_chunks(k, mode):
    """Rows of k entries and one entry less and more (up to twelve per chunk)."""
    rng = np.random.default_rng(k)
    net = _from_degrees(k + rng.integers(-1, 2, 1500), 40, k)
    ref = _per_step(LeviathanEngine(*net.engine_args(), math_mode=mode))
    want_r = ref.step_n(DT, 30)
    want = _state(ref)
    ref.close()
    e = LeviathanEngine(*net.engine_args(), math_mode=mode)
    e.set_cluster_mode(False)
    e.set_grid_mode(True, 256)
    np.testing.assert_array_equal(e.step_n(DT, 30), want_r)
    _same(_state(e), want)
    e.close()


@pytest.mark.parametrize("N,k,on", [(80_000, 24, True), (80_000, 28, False), (75_000, 28, True)])
def test_grid_kernel_is_the_default_where_its_gathers_keep_their_cache(N, k, on):
    """Three CTAs per SM with more than 64 KB of edges each are left to the
    per-step launches; the path can still be asked for."""
    net = make_network(N, k, 0.1, 9, seed=k, delay_lo=1)
    ref = _per_step(LeviathanEngine(*net.engine_args()))
    want_r = ref.step_n(DT, 12)
    want = _state(ref)
    ref.close()
    e = LeviathanEngine(*net.engine_args())
    assert e.grid_info()["eligible"] and e.grid_info()["enabled"] == on
    np.testing.assert_array_equal(e.step_n(DT, 6), want_r[:6])
    e.set_grid_mode(True)
    assert e.grid_info()["enabled"]
    np.testing.assert_array_equal(e.step_n(DT, 6), want_r[6:])
    _same(_state(e), want)
    e.close()


def _long_rows(N, seed):
    """Rows of 4 to 12 entries, and in some blocks of 256 rows one or two of 100 to
    280 among them (neighbours, so that a CTA's slices fit its shared memory):
    CTAs whose scatter takes many times that of the others.  Weights of a long
    row are scaled to those of a row of eight."""
    rng = np.random.default_rng(seed)
    deg = rng.integers(4, 13, N)
    for b in rng.choice(N // 256, max(1, N // 1500), replace=False):
        at = 256 * b + 32 * rng.integers(0, 8) + rng.integers(0, 31)
        deg[at:at + rng.integers(1, 3)] = rng.integers(100, 281)
    net = _from_degrees(deg, 30, seed)
    net.weights[:] *= np.repeat(np.minimum(1.0, 8.0 / deg), deg).astype(np.float32)
    return net


# The forward pass is bitwise; a gradient is a sum over 60 steps of sums of up to
# 280 float32 terms: sqrt(60 * 280) * 6e-8 = 8e-6 of the vector's norm on either
# side.  dL/dK, one number, cancels to a part of its terms: the bound against float64.
@pytest.mark.parametrize("N", [700, 6000, 20_000])
def test_reverse_segments_on_long_rows_among_short_ones(N):
    net = _long_rows(N, N)
    T = 60
    assert net.delays.min() >= 1
    rng = np.random.default_rng(2)
    drive = rng.normal(0, 0.5, (T, N)).astype(np.float32)
    wsel = (rng.normal(size=N) / np.sqrt(N)).astype(np.float32)

    def grads(grid, paired):
        e = LeviathanEngine(*net.engine_args(), math_mode="accurate")
        adj = Adjoint(e, segment=20, max_steps=T)
        adj.set_grid_mode(bool(grid), grid)
        adj.set_grid_pairing(paired)
        p = [torch.tensor(v, dtype=torch.float32, device="cuda", requires_grad=True)
             for v in (net.omega, net.weights, np.array([1.5]), drive)]
        r, th = simulate(adj, p[0], p[1], p[2], T, DT, drive=p[3], record_theta=True)
        ((torch.cos(th) @ torch.tensor(wsel, device="cuda")).pow(2).mean()
         + r[:, 0].mean()).backward()
        out = [r.detach().cpu().numpy(), th.detach().cpu().numpy()]
        out += [v.grad.double().cpu().numpy().ravel() for v in p]
        rows = adj.grid_info()["eligible_rows"]
        adj.close()
        e.close()
        return out, rows

    want, rows = grads(0, False)
    assert rows
    for R in rows:
        for paired in (True, False):
            got, _ = grads(R, paired)
            for a, b in zip(got[:2], want[:2]):
                np.testing.assert_array_equal(a, b)
            for name, a, b, tol in zip(("omega", "w0", "K", "drive"), got[2:], want[2:],
                                       (3e-5, 3e-5, 1e-3, 3e-5)):
                err = np.linalg.norm(a - b) / np.linalg.norm(b)
                assert err < tol, (R, paired, name, err)
    if N > 1000:
        return
    t64 = [torch.tensor(np.asarray(v, np.float64), requires_grad=True)
           for v in (net.omega, net.weights, 1.5, drive)]
    r, th = simulate64(net, t64[0], t64[1], t64[2], T, DT, drive=t64[3], record_theta=True)
    ((torch.cos(th) @ torch.tensor(wsel.astype(np.float64))).pow(2).mean() + r.mean()).backward()
    for name, a, v in zip(("omega", "w0", "K", "drive"), want[2:], t64):
        b = v.grad.numpy().ravel()
        assert np.linalg.norm(a - b) <= 1e-3 * np.linalg.norm(b), name


@pytest.mark.parametrize("N", [120_000, 200_000, 600_000])
def test_long_pair_chains_with_dependent_launches(N):
    """More than one wave of pair CTAs: blocks issued directly, recorded and
    replayed, and single steps between, bitwise as single step launches."""
    net = make_network(N, 32, 0.1, 64, seed=N, delay_lo=1)
    ref = _per_step(LeviathanEngine(*net.engine_args()))
    want_r = ref.step_n(DT, 331)
    want = _state(ref)
    ref.close()
    e = LeviathanEngine(*net.engine_args())
    e.set_grid_mode(False)
    r = [e.step_n(DT, 100), e.step_n(DT, 100)]
    r += [[e.step(DT)] for _ in range(31)]
    r += [e.step_n(DT, 100)]
    np.testing.assert_array_equal(np.concatenate(r).astype(np.float32), want_r)
    _same(_state(e), want)
    e.close()


@pytest.mark.parametrize("batch", [False, True])
def test_calls_right_after_a_single_step(batch):
    """step() returns when r has arrived; what is called next is ordered after
    the step all the same: hub counts, state, a new adjoint, close."""
    nets = [make_network(n, 8, 0.1, 20, seed=n, delay_lo=1) for n in (700, 1500)]
    for i in range(20):
        def make():
            return (BatchEngine([n.as_dict() for n in nets]) if batch
                    else LeviathanEngine(*nets[i % 2].engine_args()))
        ref = _per_step(make())
        want_r = ref.step_n(DT, 1 + i % 3)[-1]
        want = _state(ref)
        ref.close()
        e = make()
        m = HubTransitions([0, 31, 256])
        m.attach(e)
        for _ in range(1 + i % 3):
            r = e.step(DT)
        assert m.read()[3] == 1 + i % 3
        np.testing.assert_array_equal(np.float32(r), want_r)
        _same(_state(e), want)
        e.step(DT)
        e.close()
        m.close()


def test_grid_info_counts_the_ctas_of_every_network():
    sizes = (700, 64, 1500, 1)
    e = BatchEngine([make_network(n, 4, 0.1, 6, seed=n, delay_lo=1).as_dict() if n > 1
                     else _from_degrees(np.zeros(1, int), 3, 1).as_dict() for n in sizes])
    for R in e.grid_info()["eligible_rows"]:
        e.set_grid_mode(True, R)
        info = e.grid_info()
        assert info["rows_per_cta"] == R and info["ctas"] == sum(-(-n // R) for n in sizes)
    e.close()


def test_tuned_choices_reach_later_engines_together():
    """What autotune settled on, one pair variant for all classes or one per class,
    is what a later engine of the same networks starts with; networks of a class
    that was never tuned go with the tuned ones."""
    ring = [make_network(n, k, 0.1, 30, seed=n, delay_lo=1).as_dict()
            for n, k in ((90_000, 6), (61_000, 16), (70_000, 40))]

    e = BatchEngine(ring[:2])
    e.autotune(DT, 8)
    tuned = {c["cls"]: c for c in e.pair_info() if c["step_ms"] > 0.0}  # classes with networks
    assert len(tuned) == 2
    assert all(c["pair_ms"] > 0.0 for c in tuned.values())
    e.close()
    e = BatchEngine(ring[:2])
    for c in e.pair_info():
        if c["cls"] in tuned:
            assert c["pair_variant"] == tuned[c["cls"]]["pair_variant"]
    e.close()
    e = BatchEngine(ring)
    if all(c["pair_variant"] >= 0 for c in tuned.values()):
        assert ({c["pair_variant"] for c in e.pair_info()}
                <= {c["pair_variant"] for c in tuned.values()})
    want_r = None
    for per_step in (False, True):  # ... and the mixture runs as any other
        b = _per_step(BatchEngine(ring)) if per_step else e
        r = b.step_n(DT, 12)
        want_r = r if want_r is None else want_r
        np.testing.assert_array_equal(r, want_r)
        b.close()


@pytest.mark.parametrize("R", [64, 128, 256])
def test_adjoint_after_a_change_of_math_mode(R):
    """What fits of the grid-resident adjoint kernels is looked at per math mode
    when it is first needed."""
    net = make_network(3000, 10, 0.1, 20, seed=8, delay_lo=1)
    T, out = 50, []
    for mode, then in (("accurate", None), ("reference", "accurate")):
        e = LeviathanEngine(*net.engine_args(), math_mode=mode)
        adj = Adjoint(e, segment=20, max_steps=T)
        if then:
            e.set_math_mode(then)
        adj.set_grid_mode(True, R)
        info = adj.grid_info()
        assert info["enabled"] and info["rows_per_cta"] == R and info["paired"]
        assert R in info["eligible_rows"]
        p = [torch.tensor(v, dtype=torch.float32, device="cuda")
             for v in (net.omega, net.weights, np.array([1.5]))]
        r = adj.forward(*p, T, DT)
        g = adj.backward(torch.ones_like(r))
        out.append([r.cpu().numpy()] + [g[k].cpu().numpy() for k in ("omega", "w0")])
        adj.close()
        e.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.linalg.norm(a - b) < REL * np.linalg.norm(b)


# rows too long for 16 bytes of shared memory per entry at R rows per CTA, up to
# two CTAs per SM and three; bounds as for the long rows above
@pytest.mark.parametrize("N,k,R,lo,mode", [(2000, 400, 64, 1, "accurate"),
                                           (2000, 200, 128, 1, "reference"),
                                           (2001, 100, 256, 1, "accurate"),
                                           (2001, 100, 256, 0, "reference"),
                                           (19_500, 80, 64, 1, "reference")])
def test_reverse_segments_of_rows_that_fill_the_shared_memory(N, k, R, lo, mode):
    net = make_network(N, k, 0.1, 25, seed=N + k, delay_lo=lo)
    net.weights[:] *= np.float32(8.0 / k)
    T, out = 45, []
    for grid in (0, R):
        e = LeviathanEngine(*net.engine_args(), math_mode=mode)
        adj = Adjoint(e, segment=20, max_steps=T)
        assert R in adj.grid_info()["eligible_rows"]
        adj.set_grid_mode(bool(grid), grid)
        p = [torch.tensor(v, dtype=torch.float32, device="cuda")
             for v in (net.omega, net.weights, np.array([1.5]))]
        r, th = adj.forward(*p, T, DT, record_theta=True)
        g = adj.backward(torch.ones_like(r), torch.sin(th) / N)
        out.append([v.cpu().numpy() for v in (r, th, g["omega"], g["w0"])])
        adj.close()
        e.close()
    for a, b in zip(out[1][:2], out[0][:2]):
        np.testing.assert_array_equal(a, b)
    for a, b in zip(out[1][2:], out[0][2:]):
        assert np.linalg.norm(a - b) < 3e-5 * np.linalg.norm(b)


# tiles of 256 rows at the limits of the dependent launches on 148 SMs: 133 | 134,
# and one wave of each kind of pair variant (two, three, four CTAs per SM)
@pytest.mark.parametrize("tiles,variants", [(133, (4, 0)), (134, (4, 0)), (296, (6,)), (297, (6,)),
                                            (444, (4, 0)), (445, (4, 0)), (592, (4,)),
                                            (593, (4,))])
def test_pair_chain_at_the_waves_of_its_variants(tiles, variants):
    N = 256 * tiles - 3
    net = make_network(N, 4, 0.1, 7, seed=N, delay_lo=1)
    ref = _per_step(LeviathanEngine(*net.engine_args()))
    want_r = ref.step_n(DT, 21)
    want = _state(ref)
    ref.close()
    for v in variants:
        e = LeviathanEngine(*net.engine_args())
        e.set_cluster_mode(False)
        e.set_grid_mode(False)
        for c in range(3):
            e.set_pair_variant(c, v)
        r = [e.step_n(DT, 6), e.step_n(DT, 6), e.step_n(DT, 6), [e.step(DT) for _ in range(3)]]
        np.testing.assert_array_equal(np.concatenate(r).astype(np.float32), want_r)
        _same(_state(e), want)
        e.close()


# rows per CTA of an adjoint by default on 148 SMs: 14,208 rows are the last that have the paired
# backward launch at 64, 28,416 at 128; 18,944 are two CTAs of 64 per SM
@pytest.mark.parametrize("N,k,mode,segment,R,paired",
                         [(14_208, 8, "reference", 10, 64, True),
                          (14_209, 8, "reference", 10, 128, True),
                          (14_209, 8, "reference", 20, 64, False),
                          (14_209, 28, "reference", 10, 64, False),
                          (18_944, 8, "accurate", 10, 64, False),
                          (18_945, 8, "accurate", 10, 128, True),
                          (28_416, 8, "reference", 10, 128, True),
                          (28_417, 8, "reference", 10, 128, False)])
def test_adjoint_rows_per_cta(N, k, mode, segment, R, paired):
    net = make_network(N, k, 0.1, 6, seed=N, delay_lo=1)
    T, out = 20, []
    for grid in (True, False):
        e = LeviathanEngine(*net.engine_args(), math_mode=mode)
        adj = Adjoint(e, segment=segment, max_steps=T)
        info = adj.grid_info()
        assert info["enabled"] and (info["rows_per_cta"], info["paired"]) == (R, paired)
        adj.set_grid_mode(grid)
        p = [torch.tensor(v, dtype=torch.float32, device="cuda")
             for v in (net.omega, net.weights, np.array([1.5]))]
        r = adj.forward(*p, T, DT)
        g = adj.backward(torch.ones_like(r))
        out.append([r.cpu().numpy()] + [g[k].cpu().numpy() for k in ("omega", "w0")])
        adj.close()
        e.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.linalg.norm(a - b) < REL * np.linalg.norm(b)


# 20,000 rows: up to three CTAs per SM; a drive win_i x(t) without a readout
@pytest.mark.parametrize("lo,mode", [(1, "reference"), (0, "accurate")])
def test_grid_segments_with_a_lone_reservoir_drive(lo, mode):
    N, T = 20_000, 45
    net = make_network(N, 6, 0.1, 9, seed=lo, delay_lo=lo)
    rng = np.random.default_rng(5)
    win = torch.tensor(rng.normal(size=N).astype(np.float32), device="cuda")
    x = torch.tensor(rng.normal(size=(T, 1)).astype(np.float32), device="cuda")
    e = LeviathanEngine(*net.engine_args(), math_mode=mode)
    adj = Adjoint(e, segment=20, max_steps=T)
    p = [torch.tensor(v, dtype=torch.float32, device="cuda")
         for v in (net.omega, net.weights, np.array([1.5]))]
    g_win = torch.empty(N, device="cuda")
    _lib.check(adj.lib.lev_adj_set_reservoir(adj._h, win.data_ptr(), x.data_ptr(), None, None, None))
    _lib.check(adj.lib.lev_adj_set_reservoir_grads(adj._h, None, g_win.data_ptr(), None, None))
    out = {}
    for R in [0] + adj.grid_info()["eligible_rows"]:
        for paired in (True, False) if R else (False,):
            adj.set_grid_mode(bool(R), R)
            adj.set_grid_pairing(paired)
            assert adj.grid_info()["enabled"] == bool(R)
            r, th = adj.forward(*p, T, DT, record_theta=True)
            g = adj.backward(torch.ones_like(r), torch.sin(th) / N)
            out[R, paired] = [r, th, g["omega"], g["w0"], g_win.clone()]
    adj.close()
    e.close()
    want = out.pop((0, False))
    assert len(out) >= 4
    for key, got in out.items():
        for a, b in zip(got[:2], want[:2]):
            assert torch.equal(a, b), key
        for a, b in zip(got[2:], want[2:]):
            assert _rel(a, b) <= REL, key

"""Learned WENO weights on the GPU, checked against the numpy oracle of the
network (oracle/mlp_oracle.py): the training kernels' loss and gradient, the
SIMT and tensor-core evaluations (left edge and mirrored right edge), and
training on stencils harvested from the plain dycore.  Then the learned form
inside the dycore: with every stencil sent to the fallback it reproduces the
plain kernels, immersed neighbourhoods always fall back, and the trained
network's error against the FP64 build versus the untrained network's."""
import numpy as np
import pytest

import mlp_oracle as mo
from porturb_b200 import Dycore, cases
from helpers import gpu_run, twice_in_y

pytestmark = pytest.mark.gpu


def _handle(case=None):
    case = case or cases.small_mixed(immersed=False)
    g = Dycore.from_case(case, precision="f32")
    rd, u, v, w, T, trc = [np.ascontiguousarray(a) for a in case.coupler_arrays(perturbed=True)]
    g.init(rd, u, v, w, T, list(trc), None)
    return g


def _random_batch(n, seed=0):
    rng = np.random.default_rng(seed)
    x = mo.normalize(rng.normal(size=(n, 9)).cumsum(axis=1) * rng.uniform(0.1, 3, size=(n, 1)))
    z = rng.normal(size=(n, 5)) * 2
    t = np.exp(z) / np.exp(z).sum(axis=1, keepdims=True)
    return x.astype(np.float32), t.astype(np.float32)


def test_gradient_matches_numpy_oracle(gpu_lib):
    g = _handle()
    theta = g.learned_get_weights()
    assert np.allclose(theta, mo.init_params(0).astype(np.float32), rtol=1e-6, atol=1e-7)
    x, t = _random_batch(1000)
    grad, loss = g.learned_gradient(x, t)
    loss_o, grad_o = mo.loss_and_grad(theta.astype(np.float64), x, t)
    assert abs(loss - loss_o) < 1e-5 * abs(loss_o)
    rel = np.linalg.norm(grad - grad_o) / np.linalg.norm(grad_o)
    print("gradient relative L2 error vs numpy:", rel)
    assert rel < 1e-3
    for name, lo, hi in (("W1", 0, 288), ("W2", 320, 1344), ("W3", 1376, 1536), ("b3", 1536, 1541)):
        r = np.linalg.norm(grad[lo:hi] - grad_o[lo:hi]) / np.linalg.norm(grad_o[lo:hi])
        assert r < 3e-3, (name, r)


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 511, 4101])
def test_gradient_at_the_edges_of_a_block(gpu_lib, n):
    """Batches around the training block's 128 samples and its warps' 32, and
    over several rounds of the update kernel's 32 rows.  Bound: an activation
    whose sum lies within FP32 rounding of a bfloat16 boundary rounds to the
    neighbour (2^-8 of it, one of 32 in its layer) in the kernel and not in
    the FP64 oracle."""
    g = _handle()
    theta = (mo.init_params(3) * 1.2).astype(np.float32)
    g.learned_set_weights(theta)
    x, t = _random_batch(n, seed=n)
    grad, loss = g.learned_gradient(x, t)
    loss_o, grad_o = mo.loss_and_grad(theta.astype(np.float64), x, t)
    assert abs(loss - loss_o) < 1e-3 * abs(loss_o)
    assert np.linalg.norm(grad - grad_o) < 5e-3 * np.linalg.norm(grad_o)


@pytest.mark.parametrize("use_mma", [False, True])
def test_eval_matches_numpy_oracle(gpu_lib, use_mma):
    g = _handle()
    rng = np.random.default_rng(1)
    theta = (mo.init_params(5) * 1.5 + rng.normal(size=mo.N_PARAMS) * 0.05).astype(np.float32)
    g.learned_set_weights(theta)
    x, _ = _random_batch(3000, seed=2)
    wl, wr = g.learned_eval(x, use_mma=use_mma)
    ref_l = mo.forward(theta.astype(np.float64), x)["prob"]
    err = np.abs(wl - ref_l).max()
    print("max |w - numpy| (left):", err, "mma" if use_mma else "simt")
    assert err < 5e-3
    assert np.abs(wl.sum(axis=1) - 1).max() < 1e-5
    if use_mma:
        ref_r = mo.forward(theta.astype(np.float64), x[:, ::-1].copy())["prob"][:, ::-1]
        assert np.abs(wr - ref_r).max() < 5e-3


def test_training_on_harvested_stencils(gpu_lib):
    case = cases.abl_neutral(nx=64, ny=64, nz=48)
    g = _handle(case)
    g.advance(g.compute_time_step(), 10)
    g.learned_harvest(1 << 18, seed=1)
    st = g.learned_train(400, batch=8192, lr=2e-3, seed=3)
    print("training:", st)
    assert st["samples"] == 1 << 18
    assert st["loss_last"] < 0.8 * st["loss_first"]


# ---------------------------------------------------------------------------
# The learned form inside the dycore.
# ---------------------------------------------------------------------------
def _conserved_after(case, nsteps, dt, precision="f32", theta=None, threshold=None):
    g = _handle(case) if precision == "f32" else None
    if g is None:
        g = Dycore.from_case(case, precision=precision)
        rd, u, v, w, T, trc = [np.ascontiguousarray(a) for a in case.coupler_arrays(perturbed=True)]
        g.init(rd, u, v, w, T, list(trc), None)
    if theta is not None:
        if isinstance(theta, str):
            g.learned_get_weights()          # the untrained initial network
        else:
            g.learned_set_weights(theta)
        g.set_weno_mode("learned")
        g.learned_set_threshold(threshold)
    g.learned_counts()
    g.advance(dt, nsteps)
    st, tr = g.get_conserved()
    counts = g.learned_counts()
    g.close()
    return st, tr, counts


def _trained_on(case, spin_steps, dt, n=1 << 19):
    g = _handle(case)
    g.advance(dt, spin_steps)
    g.learned_harvest(n, seed=11)
    st = g.learned_train(3000, batch=16384, lr=2e-3, seed=12)
    st2 = g.learned_train(500, batch=65536, lr=5e-4, seed=13)
    theta = g.learned_get_weights()
    g.close()
    print("training:", st, st2)
    return theta


@pytest.mark.parametrize("name", ["abl_64x64x48", "bubble_64x4x32"])
def test_learned_threshold_zero_is_plain(gpu_lib, name):
    """Threshold 0 sends every stencil with a nonzero range to the plain
    limiter (and a constant stencil's edges are its value either way), so the
    fused learned kernels (queues, warp-uniform loops, z fallback lists) must
    reproduce the plain kernels."""
    case = {"abl_64x64x48": lambda: cases.abl_neutral(nx=64, ny=64, nz=48),
            "bubble_64x4x32": lambda: cases.warm_bubble(nx=64, ny=4, nz=32)}[name]()
    g = _handle(case)
    dt = g.compute_time_step()
    g.close()
    a, ta, _ = _conserved_after(case, 5, dt)
    b, tb, (nl, nf) = _conserved_after(case, 5, dt, theta="init", threshold=0.0)
    print(name, "learned/fallback stencils:", nl, nf, "exactly equal:", np.array_equal(a, b))
    assert nf > 0
    scale = np.abs(a).reshape(a.shape[0], -1).max(axis=1)
    diff = np.abs(a - b).reshape(a.shape[0], -1).max(axis=1)
    assert np.all(diff <= 1e-9 * np.maximum(scale, 1e-30)), diff
    assert np.abs(ta - tb).max() <= 1e-9 * max(np.abs(ta).max(), 1e-30)


def test_learned_fallback_near_immersed(gpu_lib):
    """Stencils with an immersed cell or a z wall within reach never use the
    network: with the threshold check off (1.0) the immersed case still falls
    back (the reference's any_immersed10 neighbourhood reaches 10 cells in
    each direction, so only cells farther from the cuboid use the network),
    and threshold 0 reproduces the plain kernels."""
    case = cases.small_mixed(nx=64, ny=32, nz=32, immersed=True)
    gp = Dycore.from_case(case, precision="f32")
    rd, u, v, w, T, trc = [np.ascontiguousarray(a) for a in case.coupler_arrays(perturbed=True)]
    gp.init(rd, u, v, w, T, list(trc), np.ascontiguousarray(case.immersed_proportion))
    dt = gp.compute_time_step()
    st0, tr0 = gp.get_conserved()
    gp.advance(dt, 3)
    a, ta = gp.get_conserved()
    gp.learned_get_weights()
    gp.set_weno_mode("learned")
    for thr, expect_learned in ((0.0, False), (1.0, True)):
        gp.set_conserved(st0, tr0)
        gp.learned_set_threshold(thr)
        gp.learned_counts()
        gp.advance(dt, 3)
        b, tb = gp.get_conserved()
        nl, nf = gp.learned_counts()
        print("threshold", thr, "learned/fallback:", nl, nf)
        assert nf > 0
        assert np.all(np.isfinite(b))
        if not expect_learned:
            scale = np.abs(a).reshape(a.shape[0], -1).max(axis=1)
            diff = np.abs(a - b).reshape(a.shape[0], -1).max(axis=1)
            assert np.all(diff <= 1e-9 * np.maximum(scale, 1e-30)), diff
        else:
            assert nl > 0
    gp.close()


@pytest.mark.parametrize("shape", [(32, 16, 20), (40, 24, 20), (64, 4, 24), (33, 17, 16)])
def test_sorted_queues(gpu_lib, shape):
    """The kernels sort a tile's (a warp's) stencils into a learned and a
    fallback queue.  With a network whose output is the ideal weights for any
    input, the learned edges are the nine-cell linear ones: on a flow that
    does not vary in z, without gravity, a step with the checks off equals the
    weno_all = False step (whose z edges are the cell values too) to the
    rounding of the softmax (1e-6 of each field's range).  With mixed queues
    every stencil is counted once, and two runs give the same bits."""
    nx, ny, nz = shape
    case = cases.small_mixed(nx=nx, ny=ny, nz=nz, immersed=False, ntr=1)
    case.options["enable_gravity"] = False
    rd, u, v, w, T, trc = [np.array(a, copy=True) for a in case.coupler_arrays(perturbed=True)]
    for a in (rd, u, v, T, trc[0]):
        a[...] = a[nz // 2]
    w[...] = 0.0
    theta = np.zeros(mo.N_PARAMS, np.float32)
    theta[-5:] = np.log(np.array([5, 40, 60, 20, 1]) / 126)

    def step(threshold, weno_all=True):
        o = dict(case.options, weno_all=weno_all)
        g = Dycore(nx, ny, nz, 100.0, 100.0, 100.0, case.tracers, o)
        g.init(rd, u, v, w, T, [trc[0]], None)
        if threshold is not None:
            g.learned_set_weights(theta)
            g.set_weno_mode("learned")
            g.learned_set_threshold(threshold)
        g.learned_counts()
        g.advance(g.compute_time_step(), 1)
        st, _ = g.get_conserved()
        counts = g.learned_counts()
        g.close()
        return st, counts

    lin, _ = step(None, weno_all=False)
    st, (nl, _) = step(2.0)
    assert nl > 0
    for a, b in zip(st, lin):
        assert np.abs((a - b)[6:nz - 6]).max() <= 1e-6 * max(np.abs(b).max(), 1e-30)
    a, ca = step(0.4)
    b, cb = step(0.4)
    assert ca == cb and ca[0] > 0 and ca[1] > 0
    assert sum(ca) == sum(step(0.0)[1]) == sum(step(2.0)[1])
    assert np.array_equal(a, b)


@pytest.mark.parametrize("nx,ny,nz,ntr,immersed", [(64, 8, 20, 1, False), (64, 8, 33, 3, True), (32, 12, 20, 4, True)])
def test_mixed_queues_do_not_depend_on_the_tile(gpu_lib, nx, ny, nz, ntr, immersed):
    """The same flow repeated once more in y goes through the 16x16 x/y tiles
    instead of the 32x4 ones and through other warps of the z march, with other
    queues; a stencil's edges are its own, so each copy has the bits of the
    flow by itself, and every stencil of it takes the same kind of weights."""
    one = cases.small_mixed(nx=nx, ny=ny, nz=nz, ntr=ntr, immersed=immersed)
    cells = gpu_run(one, "f32", 0, 0.0)[2].get_hydrostasis()[0]
    runs = []
    for case in (one, twice_in_y(one)):
        g = gpu_run(case, "f32", 0, 0.0, hydro=cells)[2]
        g.learned_set_weights((mo.init_params(3) * 0.7).astype(np.float32))
        g.set_weno_mode("learned")
        g.learned_set_threshold(0.4)
        g.learned_counts()
        g.advance(0.5 * g.compute_time_step(), 2)
        runs.append(g.get_conserved() + g.learned_counts())
        g.close()
    (sa, ta, la, fa), (sb, tb, lb, fb) = runs
    assert la > 0 and fa > 0 and np.isfinite(sa).all()
    for a, b in ((sa, sb), (ta, tb)):
        assert np.array_equal(a, b[:, :, :ny]) and np.array_equal(a, b[:, :, ny:])


def test_learned_modes_rejected_where_unsupported(gpu_lib):
    case = cases.small_mixed(immersed=False)
    g64 = Dycore.from_case(case, precision="f64")
    with pytest.raises(Exception):
        g64.set_weno_mode("learned")
    g64.close()
    g = Dycore.from_case(case, precision="f32")
    with pytest.raises(Exception):
        g.set_weno_mode("learned")      # no trained or loaded weights yet
    g.close()


def test_trained_network_gain_vs_fp64(gpu_lib):
    """Warm bubble 64x4x32, 60 steps, errors against the FP64 build.

    * The gain of training: the FP32 run with learned weights stays close to
      the FP64 build (momentum and rho*theta within 2e-3 of the field scale)
      and is several times more accurate than the same kernels with the
      untrained network (measured on a B200: 4x-10x for rho*u, rho*w and
      rho*theta).
    * Against the method without the network (the plain limiter) there is no
      gain: the plain FP32 run is more accurate (measured 1.4e-5 / 4.2e-5 /
      1.3e-4 for rho*u / rho*w / rho*theta against the learned form's 7.1e-4 /
      6.5e-4 / 8.5e-4) and faster (the bench's `learned` object).  The
      learned form's error is bounded here at 100x the plain form's, so that a
      regression of the learned form shows."""
    case = cases.warm_bubble(nx=64, ny=4, nz=32)
    g = _handle(case)
    dt = g.compute_time_step()
    g.close()
    theta = _trained_on(case, 30, dt)
    ref, _, _ = _conserved_after(case, 60, dt, precision="f64")
    plain, _, _ = _conserved_after(case, 60, dt)
    lrn, _, (nl, nf) = _conserved_after(case, 60, dt, theta=theta, threshold=0.5)
    unt, _, _ = _conserved_after(case, 60, dt, theta="init", threshold=0.5)

    def err(x):
        out = []
        for q in range(5):
            dev = ref[q] - ref[q].mean(axis=(1, 2), keepdims=True)
            scale = max(np.sqrt(np.mean(dev ** 2)), 1e-30)
            out.append(np.sqrt(np.mean((x[q] - ref[q]) ** 2)) / scale)
        return np.array(out)

    e_plain, e_lrn, e_unt = err(plain), err(lrn), err(unt)
    print("rel L2 vs FP64 (rho, rhou, rhov, rhow, rhotheta)\n plain  ", e_plain, "\n learned", e_lrn,
          "\n untrained", e_unt, "\n learned/fallback stencils", nl, nf)
    assert nl > 0
    for q in (1, 3, 4):
        assert e_lrn[q] < 2e-3
        assert e_lrn[q] < 0.35 * e_unt[q]
        assert e_lrn[q] < 100 * e_plain[q]

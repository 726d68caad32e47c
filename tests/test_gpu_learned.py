"""The learned coarse-grid correction on the GPU.

* forward and MSE-loss gradients of the CUDA network kernels against the CPU
  oracle (oracle/learned.py) on the same parameters and inputs;
* the energy-loss training path (solver-bound, level-2 Galerkin operator)
  against central finite differences of its own loss;
* training lowers the energy loss;
* what the trained network gains over the plain V-cycle: solves with it
  attached converge to the same solution, and the auto mode measures both
  and keeps the plain V-cycle whenever the network does not lower the
  iteration count.
"""
import json
import os
import sys
import time

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))
import learned  # noqa: E402

pytestmark = pytest.mark.gpu


def _f32(a):
    import torch
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float32).reshape(-1), device="cuda")


def test_forward_matches_oracle(gputo):
    import torch
    rng = np.random.default_rng(1)
    dims = (6, 5, 7)
    th = learned.init_params(2)
    th[learned.num_params() - 3:] = [0.1, -0.2, 0.3]    # nonzero output bias
    x = rng.standard_normal((4,) + dims).astype(np.float32)
    net = gputo.Net(seed=0)
    net.set_params(th)
    y = torch.empty(3 * np.prod(dims), dtype=torch.float32, device="cuda")
    net.forward(_f32(x), dims, y)
    ref, _ = learned.forward(x, th)
    got = y.cpu().numpy().reshape(ref.shape)
    assert np.abs(got - ref).max() <= 1e-4 * np.abs(ref).max()


def test_mse_gradient_matches_oracle(gputo):
    rng = np.random.default_rng(2)
    dims = (5, 4, 6)
    th = learned.init_params(4)
    xs = rng.standard_normal((2, 4) + dims).astype(np.float32)
    ts = rng.standard_normal((2, 3) + dims).astype(np.float32)
    ms = (rng.random((2, 3) + dims) > 0.3).astype(np.float32)
    net = gputo.Net(seed=0)
    net.set_params(th)
    g = np.zeros(learned.num_params(), dtype=np.float32)
    loss = net.train_step(_f32(xs), _f32(ts), _f32(ms), 2, dims, 0.0, grads_out=g)
    ref_g = np.zeros(learned.num_params())
    ref_l = 0.0
    for q in range(2):
        y, acts = learned.forward(xs[q], th)
        l, gy = learned.loss(y, ts[q], ms[q])
        ref_l += l / 2
        ref_g += learned.backward(acts, th, gy)
    assert abs(loss - ref_l) <= 1e-4 * abs(ref_l)
    assert np.abs(g - ref_g).max() <= 1e-3 * np.abs(ref_g).max()
    # the step with lr = 0 left the parameters alone
    assert np.array_equal(net.get_params(), th)


@pytest.mark.parametrize("dims,ns", [((1, 1, 1), 1), ((2, 1, 2), 257), ((3, 2, 129), 2), ((7, 12, 31), 3), ((4, 40, 1), 2)])
def test_tiles_and_samples_match_oracle(gputo, dims, ns):
    """Forward and gradients where the 128-row tiles and the stacked samples can
    go wrong: grids smaller than a tile, lines longer than one, single lines and
    planes, tiles that end inside a line, and more samples than one pass takes.
    Sums of up to 864 products in FP32: 864 2^-24 = 5e-5 of the largest, within
    the tolerances of the tests above."""
    import torch
    rng = np.random.default_rng(int(np.prod(dims)) + ns)
    th = learned.init_params(3)
    th[learned.num_params() - 3:] = [0.1, -0.2, 0.3]
    xs = rng.standard_normal((ns, 4) + dims).astype(np.float32)
    ts = rng.standard_normal((ns, 3) + dims).astype(np.float32)
    ms = (rng.random((ns, 3) + dims) > 0.3).astype(np.float32)
    net = gputo.Net(seed=0)
    net.set_params(th)
    y = torch.empty(3 * int(np.prod(dims)), dtype=torch.float32, device="cuda")
    net.forward(_f32(xs[0]), dims, y)
    ref, _ = learned.forward(xs[0], th)
    assert np.abs(y.cpu().numpy().reshape(ref.shape) - ref).max() <= 1e-4 * np.abs(ref).max()
    g = np.zeros(learned.num_params(), dtype=np.float32)
    loss = net.train_step(_f32(xs), _f32(ts), _f32(ms), ns, dims, 0.0, grads_out=g)
    ref_g, ref_l = np.zeros(learned.num_params()), 0.0
    for q in range(ns):
        yq, acts = learned.forward(xs[q], th)
        l, gy = learned.loss(yq, ts[q], ms[q])
        ref_l += l / ns
        ref_g += learned.backward(acts, th, gy)
    assert abs(loss - ref_l) <= 1e-4 * abs(ref_l)
    assert np.abs(g - ref_g).max() <= 1e-3 * np.abs(ref_g).max()


@pytest.mark.parametrize("dims,ns", [((7, 12, 31), 40), ((16, 15, 14), 9), ((3, 2, 129), 23)])
def test_weight_gradients_of_stacked_samples_are_the_sums(gputo, dims, ns):
    """A pass over many samples, where a block takes several chunks of row tiles
    (the last one short), gives the sum of the samples' own gradients, which
    take one or two chunks each.  Activations and their masks are the same bits
    on both sides.  A chunk of 512 rows is at most 32 truncating FP32 adds, 4e-6
    of its sum; for random terms that is 4e-6 sqrt(rows / 512) of the total if
    all chunks err the same way, and as much again for the separate passes."""
    rng = np.random.default_rng(int(np.prod(dims)) + ns)
    th = learned.init_params(5)
    xs = rng.standard_normal((ns, 4) + dims).astype(np.float32)
    ts = rng.standard_normal((ns, 3) + dims).astype(np.float32)
    ms = np.ones((ns, 3) + dims, dtype=np.float32)
    net = gputo.Net(seed=0)
    net.set_params(th)
    g, one = (np.zeros(learned.num_params(), dtype=np.float32) for _ in range(2))
    net.train_step(_f32(xs), _f32(ts), _f32(ms), ns, dims, 0.0, grads_out=g)
    ref = np.zeros(learned.num_params())
    for q in range(ns):
        net.train_step(_f32(xs[q:q + 1]), _f32(ts[q:q + 1]), _f32(ms[q:q + 1]), 1, dims, 0.0, grads_out=one)
        ref += one
    tol = 2 * 4e-6 * np.sqrt(ns * np.prod([d + 1 for d in dims]) / 512)
    o = 0
    for ci, co, k in ((4, 16, 27), (16, 32, 27), (32, 64, 27), (64, 3, 1)):
        for n in (ci * co * k, co):
            assert np.abs(g[o:o + n] - ref[o:o + n]).max() <= tol * np.abs(ref[o:o + n]).max()
            o += n
    assert o == g.size


@pytest.mark.parametrize("dims,ns", [((7, 6, 9), 2), ((5, 1, 3), 3)])
def test_training_keeps_the_order_of_its_sums(gputo, dims, ns):
    """A training amplifies the last bit of a gradient (Adam divides it by its own size, the weights are rounded to
    BF16), so the gradients of every step of one are pinned bit for bit to the FP32 sums in their order: more nodes
    than a CTA has threads, and fewer."""
    rng = np.random.default_rng(int(np.prod(dims)))
    xs = rng.standard_normal((ns, 4) + dims).astype(np.float32)
    ts = rng.standard_normal((ns, 3) + dims).astype(np.float32)
    ms = (rng.random((ns, 3) + dims) > 0.3).astype(np.float32)
    net = gputo.Net(seed=0)
    th = learned.init_params(11)
    th[-3:] = [0.1, -0.2, 0.3]
    net.set_params(th)
    for step in range(4):
        ref = learned.train_gradients_fp32(xs, ts, ms, net.get_params())
        g = np.zeros(learned.num_params(), dtype=np.float32)
        net.train_step(_f32(xs), _f32(ts), _f32(ms), ns, dims, 1e-3, grads_out=g)
        assert np.array_equal(g, ref), (step, np.abs(g - ref).max(), np.abs(ref).max())


def _problem(gputo, shape=(64, 32, 32), nl=4, seed=0):
    import torch
    F, fixed = gputo.cantilever(*shape)
    x = gputo.random_field_density(*shape, seed=seed, corr_len=6.0)
    CX = torch.as_tensor(1e-9 + x ** 3 * (1 - 1e-9), dtype=torch.float64, device="cuda")
    s = gputo.Solver(*shape, nl, gputo.default_options(precision=gputo.PREC_MIXED))
    s.set_problem(gputo.hex8_stiffness(), fixed)
    s.setup(CX)
    return s, torch.as_tensor(F, dtype=torch.float64, device="cuda")


def test_energy_loss_gradient_matches_finite_differences(gputo):
    """Biases enter the network in FP32 (weights are BF16-rounded), so central
    differences in every layer's biases check the energy-loss gradient through
    the whole backward pass."""
    import torch
    s, F = _problem(gputo)
    samples = gputo.harvest_net_samples(s, F, iters=3)
    X = torch.stack([q[0] for q in samples[:2]]).contiguous()
    G = torch.stack([q[1] for q in samples[:2]]).contiguous()
    net = gputo.Net(seed=5)
    th = net.get_params()
    g = np.zeros_like(th)
    s.net_train_step(net, X, G, 2, 0.0, grads_out=g)
    offs, o = [], 0
    for ws, bs in learned.layer_shapes():
        o += int(np.prod(ws))
        offs += [o + c for c in range(min(bs[0], 4))]
        o += bs[0]
    for i in offs:
        h = 1e-3
        tp, tm = th.copy(), th.copy()
        tp[i] += h
        tm[i] -= h
        net.set_params(tp)
        lp = s.net_train_step(net, X, G, 2, 0.0) * 2
        net.set_params(tm)
        lm = s.net_train_step(net, X, G, 2, 0.0) * 2
        fd = (lp - lm) / (2 * h)
        assert abs(fd - g[i]) <= 2e-2 * max(abs(fd), abs(g[i])) + 1e-3 * np.abs(g).max(), (i, fd, g[i])
    net.set_params(th)


def test_training_lowers_energy_loss(gputo):
    s, F = _problem(gputo)
    samples = gputo.harvest_net_samples(s, F, iters=20)
    net = gputo.Net(seed=1)
    hist = gputo.train_net(s, net, samples, epochs=8, lr=1e-3, batch=4)
    assert hist[-1] < hist[0] and hist[-1] < 0.0   # 0 = the plain V-cycle


def test_learned_correction_gain_and_fallback(gputo, tmp_path):
    """Train on one design, then solve a held-out design: plain, with the
    network always on, and in auto mode.  The solution is the same in all
    three; auto mode ends on whichever needed fewer iterations."""
    import torch
    s0, F = _problem(gputo, seed=0)
    samples = gputo.harvest_net_samples(s0, F, iters=30)
    net = gputo.Net(seed=1)
    gputo.train_net(s0, net, samples, epochs=4, lr=3e-4, batch=8)
    s, F = _problem(gputo, seed=11)
    res = {}
    U0 = torch.zeros_like(F)
    res["plain"] = s.solve(F, U0, 1e-8, 400)
    s.set_net(net, 1)
    U1 = torch.zeros_like(F)
    res["net"] = s.solve(F, U1, 1e-8, 400)
    assert res["net"][0] < 1e-8, res
    c0 = float(F @ U0)
    assert abs(float(F @ U1) - c0) <= 1e-6 * abs(c0)
    s.set_net(net, 2)
    nits = []
    for _ in range(4):
        U = torch.zeros_like(F)
        rr, nit = s.solve(F, U, 1e-8, 400)
        assert rr < 1e-8 and abs(float(F @ U) - c0) <= 1e-6 * abs(c0)
        nits.append(nit)
    on, plain_nit, net_nit = s.net_state()
    assert plain_nit == res["plain"][1] and net_nit == res["net"][1]
    assert on == (net_nit < plain_nit)
    assert nits[-1] == min(plain_nit, net_nit)
    gain = {"plain_nit": plain_nit, "net_nit": net_nit, "auto_uses_net": on,
            "gain_iterations": plain_nit - net_nit}
    (tmp_path / "learned_gain.json").write_text(json.dumps(gain))
    print("learned correction:", gain)


def test_attaching_another_network_replaces_the_captured_one(gputo):
    """Solves run captured iterations: after a second network is attached in the first one's place, they are those of a
    solver that only ever had the second (8 iterations, bit for bit)."""
    import torch
    nets = [gputo.Net(seed=q) for q in (1, 2)]

    def run(s, F):
        U = torch.zeros_like(F)
        return s.solve(F, U, 1e-30, 8), U

    s, F = _problem(gputo, (32, 16, 16), 3)
    s.set_net(nets[0], 1)
    (r0, n0), U0 = run(s, F)
    s.set_net(nets[1], 1)
    (r1, n1), U1 = run(s, F)
    s2, _ = _problem(gputo, (32, 16, 16), 3)
    s2.set_net(nets[1], 1)
    (r2, n2), U2 = run(s2, F)
    assert (r1, n1) == (r2, n2) and torch.equal(U1, U2)
    assert not torch.equal(U0, U1)


def test_networks_beyond_the_page_of_flags(gputo):
    """More networks at a time than the process keeps flags for: each reports its own failed pass, and none of the
    others, also where a flag has had another owner."""
    import torch
    dims, n = (3, 4, 5), 60
    x = torch.as_tensor(np.random.default_rng(1).standard_normal(4 * n), dtype=torch.float32, device="cuda")
    ok, y = (torch.empty(3 * n, dtype=torch.float32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    for count in (1030, 3):
        nets = [gputo.Net(seed=5) for _ in range(count)]
        for net in nets:
            net.forward(x, dims, ok)
        for net in (nets[0], nets[-1]):
            gputo.debug_set_sweep_fault(skip_stage=0, wait_us=200)
            try:
                with pytest.raises(gputo.GputoError) as e:
                    net.forward(x, dims, y)
                assert e.value.status == gputo.GPUTO_ERR_TIMEOUT
            finally:
                gputo.debug_set_sweep_fault(-1, 0)
            for other in (nets[1], nets[-2], net):
                other.forward(x, dims, y)
                assert torch.equal(y, ok)
        for net in nets:
            net.close()


def test_first_pass_of_a_small_network(gputo):
    """A new network's first pass on a small grid allocates once: less than half of what making the network takes (as
    long as that, and longer, when it allocates host memory that the device can write)."""
    import torch
    dims, n = (9, 9, 9), 729
    x, y = (torch.rand(c * n, device="cuda") for c in (4, 3))
    torch.cuda.synchronize()
    made, first = [], []
    for _ in range(12):
        t = [time.perf_counter()]
        net = gputo.Net(seed=6)
        t.append(time.perf_counter())
        net.forward(x, dims, y)
        t.append(time.perf_counter())
        net.close()
        made.append(t[1] - t[0])
        first.append(t[2] - t[1])
    assert np.median(first) <= 0.5 * np.median(made)

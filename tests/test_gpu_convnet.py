"""Learned-correction network: forward and backward kernels (CUDA-core and
tcgen05) against the torch-CPU oracle, and training on PM-generated pairs."""
import numpy as np
import pytest

from oracle import convnet_ref as CR

pytestmark = pytest.mark.gpu


def _net(n, seed=3):
    from cola_halo_b200.learned import ConvNet
    net = ConvNet(n, seed)
    # non-trivial biases and a larger output layer than the initialisation
    p = net.params()
    rng = np.random.default_rng(seed)
    for l in range(3):
        b0 = l * CR.LAYER + CR.WSZ
        p[b0: b0 + (16 if l < 2 else 3)] = rng.normal(0, 0.1, 16 if l < 2 else 3)
    w2 = 2 * CR.LAYER
    p[w2: w2 + CR.WSZ] *= 10
    net.set_params(p)
    return net, p


def _inputs(n, seed=5):
    rng = np.random.default_rng(seed)
    return rng.normal(0, 1, (n, n, n, 2)).astype(np.float32)


def test_forward_simt_matches_oracle(gpu_lib):
    n = 32
    net, p = _net(n)
    net.tensor_cores(False)
    x = _inputs(n)
    got = net.forward_host(x)
    want = CR.forward(x, p)[0].detach().numpy()
    err = np.abs(got - want).max() / np.abs(want).max()
    assert err < 1e-2, err          # bf16 hidden activations round at different points
    assert np.corrcoef(got.ravel(), want.ravel())[0, 1] > 0.9999


def test_backward_matches_oracle(gpu_lib):
    n = 32
    net, p = _net(n)
    net.tensor_cores(False)
    x = _inputs(n)
    g3 = np.random.default_rng(8).normal(0, 1, (n, n, n, 3)).astype(np.float32)
    got = net.backward_host(x, g3)
    want = CR.grads(x, p, g3)
    live = want != 0
    cos = np.dot(got[live], want[live]) / np.linalg.norm(got[live]) / np.linalg.norm(want[live])
    rel = np.linalg.norm(got[live] - want[live]) / np.linalg.norm(want[live])
    assert cos > 0.9999 and rel < 2e-2, (cos, rel)
    # masked weights (unused channels) get no gradient to speak of
    assert np.abs(got[~live]).max() <= 1e-3 * np.abs(got[live]).max()


def test_tensor_core_conv_matches_cuda_core(gpu_lib):
    """tcgen05 implicit-GEMM convolution (128-voxel tiles) vs the CUDA-core
    kernel on the same bf16 inputs: forward outputs and parameter gradients."""
    n = 128
    net, p = _net(n)
    x = _inputs(n, 11)
    g3 = np.random.default_rng(9).normal(0, 1, (n, n, n, 3)).astype(np.float32)
    net.tensor_cores(True)
    out_tc = net.forward_host(x)
    gr_tc = net.backward_host(x, g3)
    net.tensor_cores(False)
    out_s = net.forward_host(x)
    gr_s = net.backward_host(x, g3)
    assert np.abs(out_tc - out_s).max() <= 2e-2 * np.abs(out_s).max()
    assert np.corrcoef(out_tc.ravel(), out_s.ravel())[0, 1] > 0.99999
    rel = np.linalg.norm(gr_tc - gr_s) / np.linalg.norm(gr_s)
    assert rel < 1e-2, rel
    # and against the oracle on a slab (forward only; the oracle is O(N^3))
    want = CR.forward(x, p, dtype=__import__("torch").float32)[0].numpy()
    assert np.abs(out_tc - want).max() <= 2e-2 * np.abs(want).max()


def test_training_on_pm_pairs_reduces_force_error(gpu_lib, bbks_table):
    """Pairs from the method itself: factor-1 (coarse) vs factor-3 (fine) PM
    forces on the same particles.  After training, the corrected coarse
    force is closer to the fine force on held-out particles than the plain
    coarse force is."""
    from cola_halo_b200 import Simulation
    from cola_halo_b200.learned import ConvNet, copy_particles
    from cola_halo_b200.schedule import Schedule
    from tests.helpers import lattice_particles
    nc, L, om = 32, 100.0, 0.273
    sched = Schedule.linear(0.1, 1.0, 6)
    fine = Simulation(nc, 3 * nc, L, om)
    coarse = Simulation(nc, nc, L, om)
    net = ConvNet(nc, seed=1)
    net.set_scales(1.0, 1.0, 1.0)

    def trajectory(seed):
        p = lattice_particles(nc, L, seed, om, sched.a_init, bbks_table)
        fine.set_particles(p, sched.a_init, sched.a_init)
        states = []
        for i in range(1, sched.nloop):
            _, _, avel1, apos1 = sched.times(i)
            fine.move()
            fine.forces()
            states.append(fine.get_particles())
            fine.kick(avel1)
            fine.drift(apos1)
        return states

    train = trajectory(1) + trajectory(2)
    test = trajectory(3)[-2:]
    losses = []
    for epoch in range(40):
        for s in train:
            fine.set_particles(s, 0.5, 0.5)
            copy_particles(coarse, fine)
            losses.append(net.train_step(coarse, fine, 3e-3))
    assert np.mean(losses[-len(train):]) < 0.5 * np.mean(losses[:len(train)])

    def errs(s):
        fine.set_particles(s, 0.5, 0.5)
        fine.forces()
        ff = fine.get_forces()
        copy_particles(coarse, fine)
        coarse.forces()
        fc = coarse.get_forces()
        net.forces(coarse)
        fl = coarse.get_forces()
        return (np.sqrt(np.mean((fc - ff) ** 2)), np.sqrt(np.mean((fl - ff) ** 2)))
    for s in test:
        e_plain, e_learned = errs(s)
        assert e_learned < 0.9 * e_plain, (e_plain, e_learned)


def test_line_ring_conv_bit_identical(gpu_lib):
    """The sweep (variant 2, the default) adds the products of an output in the
    order of the kernels that take one tile at a time (two stages, one stage), in
    all three layers as a training step runs them: forward outputs are
    bit-identical.  The parameter gradients agree to the rounding of the weight
    gradient's float atomics, whose order varies from run to run."""
    from cola_halo_b200.learned import ConvNet
    n = 128
    rng = np.random.default_rng(5)
    x = rng.normal(0, 1, (n, n, n, 2)).astype(np.float32)
    g = rng.normal(0, 1, (n, n, n, 3)).astype(np.float32)
    net = ConvNet(n, seed=3)
    out, grads = [], []
    try:
        for v in (1, 2, 0, -1):
            assert gpu_lib.cg_net_set_conv_variant(v) == 0
            out.append(net.forward_host(x))
            grads.append(net.backward_host(x, g))
    finally:
        gpu_lib.cg_net_set_conv_variant(-1)
    for o, d in zip(out[1:], grads[1:]):
        np.testing.assert_array_equal(out[0], o)
        np.testing.assert_allclose(grads[0], d, rtol=1e-4, atol=1e-6 * np.abs(grads[0]).max())
    assert gpu_lib.cg_net_set_conv_variant(5) != 0
    net.close()


@pytest.mark.parametrize("n", [16, 48, 128, 144])
def test_tensor_core_weight_gradient(gpu_lib, n):
    """The tensor-core weight gradient of the last layer against float64, on
    meshes of one and of two z runs per line and with remainders of 16.  The
    first two layers are set to exact copies (powers of two of non-negative
    bf16 inputs), so the last layer's input is known bit for bit.  A weight's
    sums take at most 2 x 8 tensor-core steps in a run, one addition per run of a
    CTA and one atomic per CTA; their errors, at most 2^-23 of a partial sum whose
    terms have random signs, add up as the root of their number: 8 times that, of
    the 2-norm of the terms, leaves the largest of the 1296 weights room and is 50
    times less than g in single bf16 terms would be off.  A bias adds up to four
    gradients of a run in float32, the rest in double, then nine warps and up to
    592 CTAs in float32."""
    from cola_halo_b200.learned import ConvNet
    rng = np.random.default_rng(n)
    net = ConvNet(n, seed=1)
    p = np.zeros(net.nparams, dtype=np.float32)
    w = p.reshape(3, CR.LAYER)[:, : CR.WSZ].reshape(3, 27, 16, 16)
    for c in range(16):
        w[0, 13, c % 2, c] = 2.0 ** -(c // 2)
        w[1, 13, c, c] = 1.0
    net.set_params(p)
    x = CR.bf16(rng.uniform(0, 1, (n, n, n, 2)).astype(np.float32)).numpy()
    g = (rng.normal(0, 1, (n, n, n, 3)) * 10.0 ** rng.uniform(-6, 0, (n, n, n, 1))).astype(
        np.float32)
    got = net.backward_host(x, g).reshape(3, CR.LAYER)[2].astype(np.float64)
    net.close()
    act = np.concatenate([x.astype(np.float64) * 2.0 ** -k for k in range(8)], axis=-1)
    act, g64 = act.reshape(n, n, n, 16), g.astype(np.float64)
    runs = n * n * -(-n // 128)
    ctas = 2 * 148
    tol = 8 * np.sqrt(16 + -(-runs // ctas) + min(runs, ctas)) * 2.0 ** -23
    for t in range(27):
        a = np.roll(act, (1 - t // 9, 1 - t // 3 % 3, 1 - t % 3), axis=(0, 1, 2)).reshape(-1, 16)
        want = a.T @ g64.reshape(-1, 3)
        size = np.sqrt((a * a).T @ (g64 * g64).reshape(-1, 3))
        d = got[: CR.WSZ].reshape(27, 16, 16)[t]
        assert (np.abs(d[:, :3] - want) <= tol * size).all(), t
        assert (d[:, 3:] == 0).all()
    db = got[CR.WSZ:]
    size = np.abs(g64).sum(axis=(0, 1, 2))
    assert (np.abs(db[:3] - g64.sum(axis=(0, 1, 2))) <= (4 + 9 + 592) * 2.0 ** -24 * size).all()
    assert (db[3:] == 0).all()


def test_conv_sweep_two_tiles_per_line(gpu_lib):
    """At 256^3 a line has two tiles of 128 voxels and a CTA's run of rows
    crosses columns: the sweep's outputs are bit for bit those of one tile at
    a time."""
    from cola_halo_b200.learned import ConvNet
    n = 256
    x = np.random.default_rng(6).normal(0, 1, (n, n, n, 2)).astype(np.float32)
    net = ConvNet(n, seed=3)
    out = []
    try:
        for v in (1, 2):
            assert gpu_lib.cg_net_set_conv_variant(v) == 0
            out.append(net.forward_host(x))
    finally:
        gpu_lib.cg_net_set_conv_variant(-1)
        net.close()
    np.testing.assert_array_equal(out[0], out[1])


@pytest.mark.parametrize("n,taps", [(128, (0, 13, 26)), (128, (2, 9, 20)), (256, (6, 17, 24))])
def test_first_layer_taps(gpu_lib, n, taps):
    """Weights that pick one tap and channel each (tile and line ends, all three
    periodic faces) give the shifted inputs back exactly, the other layers
    passing them on."""
    net, p = _net(n)
    p = np.zeros_like(p)
    w = p.reshape(3, CR.LAYER)[:, :CR.WSZ].reshape(3, 27, 16, 16)
    for c, t in enumerate(taps):
        w[0, t, c % 2, c] = w[1, 13, c, c] = w[2, 13, c, c] = 1.0
    net.set_params(p)
    net.tensor_cores(True)
    # whole numbers below 256 are bf16 values; no channel is ever negative
    x = np.random.default_rng(n).integers(0, 256, (n, n, n, 2)).astype(np.float32)
    got = net.forward_host(x)
    for c, t in enumerate(taps):
        want = np.roll(x[..., c % 2], (1 - t // 9, 1 - t // 3 % 3, 1 - t % 3), axis=(0, 1, 2))
        np.testing.assert_array_equal(got[..., c], want)


@pytest.mark.parametrize("n", [16, 48, 128, 144])
def test_weight_gradients_of_every_layer_exact(gpu_lib, n):
    """All three layers' weight gradients where every partial sum is a whole
    number below 2^24, so that float32 sums are exact in any order: the layers
    pass small positive inputs through, and the output gradient is -1, 0 or 1."""
    net, p = _net(n)
    p = np.zeros_like(p)
    w = p.reshape(3, CR.LAYER)[:, :CR.WSZ].reshape(3, 27, 16, 16)
    for c in range(3):
        w[0, 13, c % 2, c] = w[1, 13, c, c] = w[2, 13, c, c] = 1.0
    net.set_params(p)
    net.tensor_cores(True)
    rng = np.random.default_rng(n)
    x = rng.integers(1, 4, (n, n, n, 2)).astype(np.float32)
    g = rng.integers(-1, 2, (n, n, n, 3)).astype(np.float32)
    got = net.backward_host(x, g).reshape(3, CR.LAYER)
    gm = g.reshape(-1, 3).astype(np.float64)
    for layer in range(3):
        chans = (0, 1) if layer == 0 else (0, 1, 0)
        want = np.zeros((27, 16, 16))
        for t in range(27):
            a = np.roll(x, (1 - t // 9, 1 - t // 3 % 3, 1 - t % 3), axis=(0, 1, 2))
            want[t, :len(chans), :3] = a.reshape(-1, 2)[:, list(chans)].T.astype(np.float64) @ gm
        np.testing.assert_array_equal(got[layer][:CR.WSZ].reshape(27, 16, 16), want, str(layer))
        np.testing.assert_array_equal(got[layer][CR.WSZ:CR.WSZ + 3], gm.sum(axis=0))


def _first_layer_only(net, w0, bias):
    """Parameters with first-layer weights w0 [27][2][3] and biases, passed on to
    the three outputs (hidden values are not negative)."""
    p = np.zeros(net.nparams, dtype=np.float32).reshape(3, CR.LAYER)
    w = p[:, :CR.WSZ].reshape(3, 27, 16, 16)
    w[0, :, :2, :3] = w0
    p[0, CR.WSZ: CR.WSZ + 3] = bias
    for c in range(3):
        w[1, 13, c, c] = w[2, 13, c, c] = 1.0
    net.set_params(p.ravel())


def test_host_forward_is_the_training_step_s(gpu_lib):
    """The host forward adds the first layer's taps one after another on every
    pipeline, as a training step does (the pairs that a force reads are added 8
    taps at a time): 2^24, 1 and -2^24 on three taps in a row give 0."""
    from cola_halo_b200.learned import ConvNet
    n = 128
    net = ConvNet(n, seed=1)
    w0 = np.zeros((27, 2, 3), dtype=np.float32)
    w0[[0, 1, 2], 0] = np.array([[2.0 ** 24], [1.0], [-2.0 ** 24]])
    _first_layer_only(net, w0, 0.0)
    x = np.ones((n, n, n, 2), dtype=np.float32)
    try:
        for v in (0, 1, 2, -1):
            assert gpu_lib.cg_net_set_conv_variant(v) == 0
            assert (net.forward_host(x) == 0).all(), v
    finally:
        gpu_lib.cg_net_set_conv_variant(-1)
        net.close()


@pytest.mark.parametrize("n", [128, 256])
def test_force_first_layer_from_packed_features(gpu_lib, n):
    """cg_net_forces reads its first layer's input as pairs on these meshes.
    Particles on mesh points give a density of whole numbers, and the output of
    their own cell: weights 0 and 1 on all taps of the density add up exactly
    (below 256, so that bf16 holds the hidden value).  A tap of the potential is
    one product, with which the CUDA-core layers, which read the 16-channel
    layout, agree exactly.  The net's output is the difference of two float
    forces: 2^-22 of the larger of them."""
    from cola_halo_b200 import PARTICLE_DTYPE, Simulation
    from cola_halo_b200.learned import ConvNet
    rng = np.random.default_rng(n)
    m = 20000
    at = np.concatenate([rng.integers(0, n, (m - 512, 3)),
                         rng.integers(0, 2, (512, 3)) * (n - 1)])       # and the corners
    p = np.zeros(m, dtype=PARTICLE_DTYPE)
    p["x"] = at
    sim = Simulation(n // 2, n, float(n), 0.273)
    sim.set_particles(p, 0.5, 0.5)
    sim.forces()
    plain = sim.get_forces().astype(np.float64)
    net = ConvNet(n, seed=1)
    net.set_scales(1.0, 1.0, 1.0)
    count = np.zeros((n, n, n))
    np.add.at(count, tuple(at.T), 8.0)           # (ngrid / nc)^3 a particle
    pick = tuple(at.T)

    def correction():
        net.forces(sim)
        return sim.get_forces().astype(np.float64) - plain

    taps = rng.integers(0, 2, (27, 3)).astype(np.float32)
    taps[[0, 13, 26]] = 1.0
    taps *= (np.cumsum(taps, axis=0) <= 8)       # at most 8 taps an output
    w0 = np.zeros((27, 2, 3), dtype=np.float32)
    w0[:, 0] = taps
    _first_layer_only(net, w0, taps.sum(axis=0))     # sum w (count - 1) + sum w
    got = correction()
    for c in range(3):
        want = sum(np.roll(count, (1 - t // 9, 1 - t // 3 % 3, 1 - t % 3), axis=(0, 1, 2))
                   for t in range(27) if taps[t, c])[pick]
        ok = want < 256
        assert ok.mean() > 0.5
        tol = 2.0 ** -22 * (np.abs(plain[:, c]) + want)
        assert (np.abs(got[:, c] - want) <= tol)[ok].all(), c
    for t0 in range(0, 27, 3):
        w0 = np.zeros((27, 2, 3), dtype=np.float32)
        for c in range(3):
            w0[t0 + c, 1, c] = 1.0
        _first_layer_only(net, w0, 0.0)
        net.tensor_cores(True)
        packed = correction()
        net.tensor_cores(False)
        wide = correction()
        assert np.abs(packed).max() > 0
        np.testing.assert_array_equal(packed, wide, str(t0))
    net.close()
    sim.close()


@pytest.mark.parametrize("n", [16, 48, 128, 144])
@pytest.mark.parametrize("layer", [0, 1, 2])
def test_weight_gradients_need_every_term(gpu_lib, n, layer):
    """Weight gradients of one layer, exact, where its output gradient is a whole
    number of 18 bits with the lowest set: rounded to one bf16 term it is another
    number, and every other one to two.  The last layer is given it; the layers below get it as the
    sum of three of six bits in steps of 2^6 (the data gradients multiply bf16
    numbers, which hold each), on all 16 channels.  Six voxels a call, at the ends of
    lines, runs and products, and inputs of 1 and 2: every partial sum is a whole
    number below 2^22."""
    rng = np.random.default_rng(100 * n + layer)
    net, p = _net(n)
    p = np.zeros_like(p)
    w = p.reshape(3, CR.LAYER)[:, :CR.WSZ].reshape(3, 27, 16, 16)
    for c in range(16):
        w[0, 13, c % 2, c] = 1.0
    if layer == 0:
        w[1, 13, :, :3] = 1.0                     # gradients of three channels, added up
        for c in range(3):
            w[2, 13, c, c] = 1.0
    else:
        w[1, 13] = np.eye(16)
        w[2, 13, :, :3] = 1.0
    net.set_params(p)
    net.tensor_cores(True)
    x = rng.integers(1, 3, (n, n, n, 2)).astype(np.float32)
    step = np.array([4096, 64, 1])
    for call in range(4):
        g = np.zeros((n, n, n, 3), dtype=np.float32)
        z = rng.permutation([0, n - 1, 15, n - 16, rng.integers(n), min(127, n - 2)])
        at = np.stack([rng.permutation(n)[:6], rng.choice([0, 1, n - 1, n // 2], 6), z], axis=1)
        parts = 2 * rng.integers(16, 32, (6, 3)) + 1          # odd, 33 .. 63
        if layer == 2:
            g[tuple(at.T)] = (2 * rng.integers(1 << 16, 1 << 17, (6, 3)) + 1) * rng.choice(
                [-1, 1], (6, 3))
        else:
            g[tuple(at.T)] = parts * step
        got = net.backward_host(x, g).reshape(3, CR.LAYER)[layer]
        # the layer's output gradient: the given one, or its channels' sum on all 16
        out = g if layer == 2 else np.repeat(g.sum(axis=-1, keepdims=True), 16, axis=-1)
        nout = out.shape[-1]
        chans = [c % 2 for c in range(2 if layer == 0 else 16)]
        dw = got[:CR.WSZ].reshape(27, 16, 16)
        for t in range(27):
            src = (at + (t // 9 - 1, t // 3 % 3 - 1, t % 3 - 1)) % n
            want = x[tuple(src.T)][:, chans].T.astype(np.float64) @ out[tuple(at.T)]
            np.testing.assert_array_equal(dw[t, :len(chans), :nout], want, str((call, t)))
        np.testing.assert_array_equal(got[CR.WSZ:CR.WSZ + nout],
                                      out.reshape(-1, nout).sum(axis=0, dtype=np.float64))
    net.close()

"""GPU checks of the learned block preconditioner through the C-ABI.

* forward, backward (parameter gradients), masked MSE and Adam of the FP32
  training kernels against the FP64 numpy oracle (oracle/unet.py), which is
  itself pinned by finite differences: 1e-4 max-norm relative per layer; the
  tensor-core training path (BF16 operands, FP32 accumulation) at BF16
  tolerances: 1e-2 on the output, 3e-2 per layer on the gradients of a
  backward from the FP32 forward's cache, cosine 0.98 for the whole BF16 pass;
* a training step is bitwise reproducible (fixed-order reductions);
* training on pairs from the context's own MGPCG solves lowers the loss;
* flexible CG preconditioned by the trained network reaches the 1e-6 relative
  FP64 residual, and an untrained network stalls and falls back to the V-cycle
  (still converging)."""

import numpy as np
import pytest

import fluidity_b200 as fb
from fluidity_b200 import learned, scenes
from helpers import dam_break_context
from oracle import unet as U

pytestmark = pytest.mark.gpu
TOL = 1e-4


def _t(a):
    import torch

    return torch.tensor(np.ascontiguousarray(a, np.float32), device="cuda")


def _rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-30))


def _inputs(rng, n):
    x = rng.normal(size=(n, 2, 10, 10, 10))
    x[:, 1] = rng.integers(-1, 2, size=(n, 10, 10, 10))
    return x


@pytest.fixture(scope="module")
def net():
    n = fb.UNet(8)
    yield n
    n.close()


def test_forward_and_backward_match_oracle(net):
    import torch

    rng = np.random.default_rng(0)
    th = U.init_params(5) + 0.02 * rng.normal(size=U.param_count())
    x = _inputs(rng, 5)
    y_ref, cache = U.forward(th, x)
    dy = rng.normal(size=y_ref.shape)
    g_ref = U.backward(th, cache, dy)
    P, X = _t(th), _t(x)
    Y = torch.zeros((5, 512), device="cuda")
    G = torch.zeros_like(P)
    net.forward(P, X, Y)
    net.backward(P, _t(dy.reshape(5, 512)), G)
    torch.cuda.synchronize()
    assert _rel(Y.cpu().numpy(), y_ref.reshape(5, 512)) <= TOL
    g = G.cpu().numpy()
    off = 0
    for name, nw, nb in U.layer_sizes():
        assert _rel(g[off:off + nw], g_ref[off:off + nw]) <= TOL, name
        assert _rel(g[off + nw:off + nw + nb], g_ref[off + nw:off + nw + nb]) <= TOL, name
        off += nw + nb


def test_tensor_core_training_matches_oracle_at_bf16_tolerance():
    """The tensor-core convolutions against the FP64 oracle.

    The forward output is checked directly. The backward is checked from the
    FP32 forward's cache, so that every ReLU mask is the oracle's: with a
    random output gradient each parameter gradient is a sum of terms of random
    sign that nearly cancel, and the few masks that a BF16 forward flips near
    zero would dominate its error. The whole BF16 forward + backward is held to
    the direction of the oracle's gradient (cosine).
    """
    import torch

    rng = np.random.default_rng(0)
    th = U.init_params(5) + 0.02 * rng.normal(size=U.param_count())
    x = _inputs(rng, 5)
    y_ref, cache = U.forward(th, x)
    dy = rng.normal(size=y_ref.shape)
    g_ref = U.backward(th, cache, dy)
    P, X, DY = _t(th), _t(x), _t(dy.reshape(5, 512))
    Y = torch.zeros((5, 512), device="cuda")
    G = torch.zeros_like(P)
    net = fb.UNet(8)
    net.forward(P, X, Y)  # FP32 forward: the oracle's masks
    net.set_tensor_cores(True)
    net.backward(P, DY, G)
    torch.cuda.synchronize()
    g = G.cpu().numpy()
    net.forward(P, X, Y)  # BF16 forward, then BF16 backward
    G2 = torch.zeros_like(P)
    net.backward(P, DY, G2)
    torch.cuda.synchronize()
    net.close()
    ey = _rel(Y.cpu().numpy(), y_ref.reshape(5, 512))
    g2 = G2.cpu().numpy()
    cos = float(g2 @ g_ref / (np.linalg.norm(g2) * np.linalg.norm(g_ref)))
    off, errs = 0, {}
    for name, nw, nb in U.layer_sizes():
        errs[name] = (_rel(g[off:off + nw], g_ref[off:off + nw]), _rel(g[off + nw:off + nw + nb], g_ref[off + nw:off + nw + nb]))
        off += nw + nb
    print(f"tensor cores vs FP64 oracle: output {ey:.2e}, full-BF16 gradient cosine {cos:.6f}, "
          f"backward per layer {({k: (round(a, 5), round(b, 5)) for k, (a, b) in errs.items()})}")
    assert ey <= 1e-2
    assert cos >= 0.98
    for name, (ew, eb) in errs.items():
        assert ew <= 3e-2 and eb <= 3e-2, (name, ew, eb)


def test_masked_mse_and_adam_match_oracle():
    import torch

    rng = np.random.default_rng(1)
    y, t = rng.normal(size=(3, 512)), rng.normal(size=(3, 512))
    m = (rng.uniform(size=(3, 512)) > 0.4).astype(np.float64)
    t[1] = 0.0  # an item without target energy
    for relative in (0, 1):
        loss_ref, grad_ref = U.masked_mse(y, t, m, relative=bool(relative))
        loss = torch.zeros(1, device="cuda")
        grad = torch.zeros((3, 512), device="cuda")
        fb.UNet.masked_mse(_t(y), _t(t), _t(m), loss, grad, relative=relative)
        assert abs(loss.item() - loss_ref) <= 1e-6 * loss_ref
        assert _rel(grad.cpu().numpy(), grad_ref) <= 1e-6
    th, gr = rng.normal(size=1000), rng.normal(size=1000)
    mm, vv = np.zeros(1000), np.zeros(1000)
    P, G, M, V = _t(th), _t(gr), _t(mm), _t(vv)
    for step in (1, 2, 3):
        th, mm, vv = U.adam(th, gr, mm, vv, step)
        fb.UNet.adam_step(P, G, M, V, step)
    np.testing.assert_allclose(P.cpu().numpy(), th, rtol=0, atol=1e-6)


def test_init_params_follow_he_uniform_rule():
    import torch

    P = torch.empty(fb.UNet.param_count(), device="cuda")
    fb.UNet.init_params(P, 7)
    p = P.cpu().numpy()
    off = 0
    for (name, kind, cin, cout), (_, nw, nb) in zip(U.LAYERS, U.layer_sizes()):
        bound = np.sqrt(6.0 / (cin * (27 if kind.startswith("conv3") else 1)))
        w = p[off:off + nw]
        assert np.all(np.abs(w) <= bound) and np.all(p[off + nw:off + nw + nb] == 0.0), name
        if nw >= 1000:
            assert abs(w.std() - bound / np.sqrt(3)) < 0.05 * bound, name
        off += nw + nb


def test_training_step_is_bitwise_reproducible():
    """Three Adam steps, twice, on the tensor-core path (the default)."""
    import torch

    rng = np.random.default_rng(2)
    x = _t(_inputs(rng, 64))
    t = _t(rng.normal(size=(64, 512)))
    m = _t((rng.uniform(size=(64, 512)) > 0.5).astype(np.float32))
    outs = []
    for _ in range(2):
        P, losses = learned.train(x, t, m, steps=3, batch=64, seed=3)
        outs.append((P.cpu().numpy(), losses))
    np.testing.assert_array_equal(outs[0][0], outs[1][0])
    np.testing.assert_array_equal(outs[0][1], outs[1][1])


@pytest.fixture(scope="module")
def trained():
    x, t, m = learned.collect_pairs(64, pairs=3000, steps_between=3, seed_steps=2, max_states=6)
    P, losses = learned.train(x, t, m, steps=1500, batch=64, seed=0)
    return x.shape[0], P, losses


def test_training_on_solver_pairs_lowers_the_loss(trained):
    """The block-residual loss |r_b - A_b y|^2 / max(|r_b|^2, 1): the zero
    correction scores at most 1; the trained network must end below half of
    that (it learns to invert the pressure operator on its block)."""
    count, P, losses = trained
    assert count >= 500
    assert np.all(np.isfinite(losses))
    assert losses[-40:].mean() < 0.5
    assert losses[-40:].mean() < 0.1 * losses[:40].mean()


def test_block_residual_loss_matches_oracle():
    import torch

    rng = np.random.default_rng(11)
    x = _inputs(rng, 5)
    x[:, 1] = rng.choice([1.0, 0.0, -1.0], p=[0.7, 0.2, 0.1], size=(5, 10, 10, 10))
    x[3, 0, 1:9, 1:9, 1:9] = 0.0  # an item without residual on its block: skipped
    y = rng.normal(size=(5, 512))
    want_loss, want_grad = U.block_residual_loss(y, x)
    loss = torch.zeros(1, device="cuda")
    grad = torch.zeros((5, 512), device="cuda")
    fb.UNet.block_residual_loss(_t(y), _t(x), loss, grad)
    assert float(loss) == pytest.approx(want_loss, rel=1e-5)
    assert _rel(grad.cpu().numpy(), want_grad) <= 1e-5
    assert np.all(grad.cpu().numpy()[3] == 0.0)


@pytest.mark.parametrize("batch", [1, 7, 8, 9, 32, 33, 128, 129, 1024])
def test_block_residual_loss_item_counts(batch):
    """Item counts around the CTAs (8) and items in flight (32) of the loss kernel. FP32 stencils of
    at most 13 terms: 1e-5; the loss and V summed in FP64; twice gives the same bits."""
    import torch

    rng = np.random.default_rng(batch)
    x = rng.normal(size=(batch, 2, 10, 10, 10)).astype(np.float32)
    x[:, 1] = rng.choice([1.0, 0.0, -1.0], p=[0.7, 0.2, 0.1], size=(batch, 10, 10, 10))
    x[batch // 2 + 1:batch // 2 + 2, 0] = 0.0  # an item without residual
    y = rng.normal(size=(batch, 512)).astype(np.float32)
    some = np.unique(np.r_[0, batch // 2, batch - 1])  # the oracle's dense operators cost 2 MB an item
    loss, grad = torch.zeros(1, device="cuda"), torch.full((batch, 512), 7.0, device="cuda")
    fb.UNet.block_residual_loss(_t(y), _t(x), loss, grad)
    again = torch.zeros_like(grad)
    fb.UNet.block_residual_loss(_t(y), _t(x), torch.zeros(1, device="cuda"), again)
    assert torch.equal(grad, again)
    want = np.zeros((batch, 512))
    total, valid = 0.0, 0
    for b in range(batch):
        if b in some or batch <= 129:
            item_loss, item_grad = U.block_residual_loss(y[b:b + 1], x[b:b + 1])
            want[b] = item_grad[0]
            total += item_loss
        valid += bool(np.any((x[b, 1] == 1.0)[1:9, 1:9, 1:9] & (x[b, 0, 1:9, 1:9, 1:9] != 0)))
    got = grad.cpu().numpy() * max(valid, 1)
    rows = some if batch > 129 else np.arange(batch)
    assert _rel(got[rows], want[rows]) <= 1e-5
    if batch <= 129:
        assert float(loss) == pytest.approx(total / max(valid, 1), rel=1e-5)


def _held_out(scene, n, steps=7):
    soa, mass = scenes.SCENES[scene](n)
    ctx = fb.LiquidContext(n, capacity=soa.shape[1])
    ctx.upload(soa)
    tp = fb.transfer_params(scenes.DT, mass)
    for _ in range(steps):
        code, _ = ctx.step(tp, fb.default_pressure_options(precision=1))
        assert code == fb.OK
    return ctx, tp


def test_trained_network_gains_over_the_vcycle_alone(trained):
    """The composite preconditioner (V-cycle, then the network's correction from
    the V-cycle's residual) on two held-out states (scenes and sizes the network
    was not trained on): never more flexible-CG iterations to the 1e-6 FP64
    residual than the V-cycle alone, and fewer on at least one; every iteration
    uses the network (no fallback). Without the network (the zero network) the
    composite is the V-cycle itself."""
    import torch

    _, P, _ = trained
    gains = []
    for scene, n in (("splash", 64), ("dam_break", 128)):
        ctx, tp = _held_out(scene, n)
        code, v = ctx.project(tp, fb.default_pressure_options(rel_tol=1e-6, warm_start=0, precision=1))
        assert code == fb.OK
        ctx.set_learned_preconditioner(torch.zeros(fb.UNet.param_count(), device="cuda"))
        code, z = ctx.project(tp, fb.default_pressure_options(rel_tol=1e-6, warm_start=0, precision=1,
                                                              preconditioner=2))
        assert code == fb.OK and z.iterations == v.iterations
        ctx.set_learned_preconditioner(P)
        code, c = ctx.project(tp, fb.default_pressure_options(rel_tol=1e-6, warm_start=0, precision=1,
                                                              preconditioner=2))
        assert code == fb.OK, c.as_dict()
        assert c.relative_residual <= 1e-6 and c.fell_back == 0 and c.learned_iterations == c.iterations
        gains.append((scene, n, v.iterations, c.iterations))
        ctx.close()
    print("V-cycle vs composite iterations:", gains)
    assert all(ci <= vi for _, _, vi, ci in gains), gains
    assert any(ci < vi for _, _, vi, ci in gains), gains


def test_learned_fcg_reaches_fp64_residual(trained):
    _, P, _ = trained
    ctx, _, m = dam_break_context(64)
    params = fb.transfer_params(scenes.DT, m)
    ctx.step(params, fb.default_pressure_options())
    ctx.set_learned_preconditioner(P)
    for prec in (0, 1):
        opt = fb.default_pressure_options(precision=prec, preconditioner=1, max_iterations=2000)
        code, d = ctx.step(params, opt)
        assert code == fb.OK, d.as_dict()
        assert d.relative_residual <= 1e-6 and d.learned_iterations > 0
    ctx.close()


def _identity_params():
    """Weights for which the network returns its residual input (z = r): a
    correction no better than plain CG."""
    P = {name: [w.copy(), b.copy()] for name, (w, b) in U.unpack(np.zeros(U.param_count())).items()}
    P["e1a"][0][0, 0, 1, 1, 1], P["e1a"][0][1, 0, 1, 1, 1] = 1.0, -1.0
    for name in ("e1b", "d1"):
        P[name][0][0, 0, 1, 1, 1] = P[name][0][1, 1, 1, 1, 1] = 1.0
    P["out"][0][0, 0], P["out"][0][0, 1] = 1.0, -1.0
    return U.pack(P)


def test_identity_network_is_exact_through_the_kernels(net):
    import torch

    rng = np.random.default_rng(4)
    x = _inputs(rng, 3)
    Y = torch.zeros((3, 512), device="cuda")
    net.forward(_t(_identity_params()), _t(x), Y)
    np.testing.assert_allclose(Y.cpu().numpy().reshape(3, 8, 8, 8), x[:, 0, 1:9, 1:9, 1:9], rtol=1e-6, atol=1e-6)


def test_tensor_core_inference_matches_fp32_forward():
    """The tcgen05 implicit-GEMM inference (BF16 activations, FP32 accumulation)
    against the FP32 training forward on the same solver windows: 3e-2 max-norm
    relative for a random network; the identity network returns r on fluid cells
    to BF16 rounding (4e-3 of max |r|)."""
    import torch

    ctx, _, m = dam_break_context(32)
    params = fb.transfer_params(scenes.DT, m)
    ctx.step(params, fb.default_pressure_options())
    nb = len(ctx.active_blocks())
    rng = np.random.default_rng(6)
    r = _t(rng.normal(size=nb * 512))
    z_tc = torch.zeros(nb * 512, device="cuda")
    z_ref = torch.zeros_like(z_tc)
    th = U.init_params(9) + 0.01 * rng.normal(size=U.param_count())
    ctx.set_learned_preconditioner(_t(th))
    ctx.apply_learned(r, z_tc, kernels=0)
    ctx.apply_learned(r, z_ref, kernels=1)
    a, b = z_tc.cpu().numpy(), z_ref.cpu().numpy()
    assert np.any(b != 0.0)
    assert _rel(a, b) <= 3e-2
    ctx.set_learned_preconditioner(_t(_identity_params()))
    ctx.apply_learned(r, z_tc, kernels=0)
    ctx.apply_learned(r, z_ref, kernels=1)
    a, b = z_tc.cpu().numpy(), z_ref.cpu().numpy()
    fluid = b != 0.0
    np.testing.assert_allclose(b[fluid], r.cpu().numpy()[fluid], rtol=1e-6, atol=1e-6)
    assert np.all(a[~fluid] == 0.0)
    assert np.abs(a - b).max() <= 4e-3 * np.abs(b).max()
    ctx.close()


def test_stalled_network_falls_back_to_the_vcycle():
    ctx, _, m = dam_break_context(32)
    params = fb.transfer_params(scenes.DT, m)
    ctx.step(params, fb.default_pressure_options())
    ctx.set_learned_preconditioner(_t(_identity_params()))
    # stall_ratio 0.01: every learned iteration counts as stalled -> fallback after exactly 3
    code, d = ctx.step(params, fb.default_pressure_options(preconditioner=1, stall_ratio=0.01))
    assert code == fb.OK
    assert d.fell_back == 1 and d.learned_iterations == 3
    assert d.relative_residual <= 1e-6
    ctx.close()


def test_zero_network_breaks_down_and_falls_back_at_once():
    import torch

    ctx, _, m = dam_break_context(32)
    params = fb.transfer_params(scenes.DT, m)
    ctx.step(params, fb.default_pressure_options())
    ctx.set_learned_preconditioner(torch.zeros(fb.UNet.param_count(), device="cuda"))  # z = 0, z.r = 0
    code, d = ctx.step(params, fb.default_pressure_options(preconditioner=1))
    assert code == fb.OK
    assert d.fell_back == 1 and d.learned_iterations == 0
    assert d.relative_residual <= 1e-6
    ctx.close()


def _open_network(seed):
    """Parameters whose every ReLU is open on _inputs: weights a tenth of the initialisation's and
    biases 1, so a layer's sum has a standard deviation of about 0.15 around at least 1. With masks
    that rounding cannot flip, the errors are those of the sums alone (one flipped mask of the 10^6
    that 40 items have moves a gradient of the first layer by 3e-3)."""
    th, off = 0.1 * U.init_params(seed), 0
    for name, nw, nb in U.layer_sizes():
        th[off + nw:off + nw + nb] = 1.0
        off += nw + nb
    return th


@pytest.mark.parametrize("batch", [1, 5, 33, 40, 160])
def test_fp32_convolutions_at_item_counts(batch):
    """The FP32 forward and backward at item counts around the items a CTA takes at 2^3 (32 in the
    convolutions, 4 in the weight gradients; one elsewhere) and, at 160, with more work units in every
    layer's weight gradient than it has CTAs (640 slabs against 296 at 8^3, 160 items against 151 and 75
    at 4^3, 40 groups against 37 at 2^3), so that CTAs take a second one; against the FP64 oracle:
    sums of at most 864 FP32 terms in the forward, 82k in a gradient, 1e-4 per layer; twice gives the
    same bits."""
    import torch

    rng = np.random.default_rng(batch)
    th = _open_network(3)
    x = _inputs(rng, batch)
    y_ref, cache = U.forward(th, x)
    dy = rng.normal(size=y_ref.shape)
    g_ref = U.backward(th, cache, dy)
    P, X, DY = _t(th), _t(x), _t(dy.reshape(batch, 512))
    Y, G, again = torch.zeros((batch, 512), device="cuda"), torch.zeros_like(P), torch.zeros_like(P)
    n = fb.UNet(batch)
    n.forward(P, X, Y)
    n.backward(P, DY, G)
    n.forward(P, X, Y)
    n.backward(P, DY, again)
    torch.cuda.synchronize()
    n.close()
    assert torch.equal(G, again)
    assert _rel(Y.cpu().numpy(), y_ref.reshape(batch, 512)) <= TOL
    g, off = G.cpu().numpy(), 0
    for name, nw, nb in U.layer_sizes():
        assert _rel(g[off:off + nw], g_ref[off:off + nw]) <= TOL, name
        assert _rel(g[off + nw:off + nw + nb], g_ref[off + nw:off + nw + nb]) <= TOL, name
        off += nw + nb


@pytest.mark.parametrize("batch", [1, 3, 17, 40, 160])
def test_tensor_core_convolutions_at_item_counts(batch):
    """The tensor-core forward, and the backward from the FP32 forward's cache, at item counts around
    the four items a CTA takes at 2^3 (one elsewhere) and, at 160, with more work units in every layer's
    weight gradient than it has CTAs (320 slabs against 148 at 8^3, 160 items against 148 and 75 at
    4^3, 40 groups against 37 at 2^3), against the FP64 oracle at BF16 tolerances (as
    test_tensor_core_training_matches_oracle_at_bf16_tolerance)."""
    import torch

    rng = np.random.default_rng(batch)
    th = _open_network(5)
    x = _inputs(rng, batch)
    y_ref, cache = U.forward(th, x)
    dy = rng.normal(size=y_ref.shape)
    g_ref = U.backward(th, cache, dy)
    P, X, DY = _t(th), _t(x), _t(dy.reshape(batch, 512))
    Y, G, again = torch.zeros((batch, 512), device="cuda"), torch.zeros_like(P), torch.zeros_like(P)
    n = fb.UNet(batch)
    n.forward(P, X, Y)
    n.set_tensor_cores(True)
    n.backward(P, DY, G)
    n.backward(P, DY, again)
    n.forward(P, X, Y)
    torch.cuda.synchronize()
    n.close()
    assert torch.equal(G, again)
    assert _rel(Y.cpu().numpy(), y_ref.reshape(batch, 512)) <= 1e-2
    g, off = G.cpu().numpy(), 0
    for name, nw, nb in U.layer_sizes():
        assert _rel(g[off:off + nw], g_ref[off:off + nw]) <= 3e-2, name
        assert _rel(g[off + nw:off + nw + nb], g_ref[off + nw:off + nw + nb]) <= 3e-2, name
        off += nw + nb


def _box_of_blocks(shape):
    """A context whose active blocks are a box of full blocks at the lattice's corner and the next layer."""
    import ctypes

    import torch

    n = 96
    axes = [(np.arange(8 * k) + 0.5) / n for k in shape]
    x = np.stack([a.ravel() for a in np.meshgrid(*axes, indexing="ij")])
    count = x.shape[1]
    soa = np.zeros((15, count), np.float32)
    soa[0:3] = x
    src, dst = _t(soa), torch.zeros((15, count), device="cuda")

    def parts(t):
        p = fb.Particles()
        p.x[:] = [t[d].data_ptr() for d in range(3)]
        p.v[:] = [t[3 + d].data_ptr() for d in range(3)]
        p.c[:] = [t[6 + d].data_ptr() for d in range(9)]
        p.mass, p.count = None, count
        return p

    ctx = fb.LiquidContext(n, capacity=count)
    lib, rep, a, b = fb.library(), fb.Report(), parts(src), parts(dst)
    assert lib.fl_topology_from_particles(ctx.handle, ctypes.byref(a), None, ctypes.byref(rep)) == fb.OK
    assert lib.fl_sort_particles_by_block(ctx.handle, ctypes.byref(a), ctypes.byref(b), None, ctypes.byref(rep)) == fb.OK
    assert len(ctx.active_blocks()) == np.prod([k + 1 for k in shape])
    return ctx


@pytest.mark.parametrize("shape", [(1, 1, 1), (6, 5, 2), (7, 3, 3), (1, 5, 10)])
def test_tensor_core_inference_at_block_counts(shape):
    """The inference where the 2^3 layer's tiles of 128 blocks end (8, 126, 128 and 132 active
    blocks: a box of full blocks at the lattice's corner and the next layer), against the FP32
    forward, with the first third of the blocks without residual: 3e-2 of the largest value, as
    the test above."""
    import torch

    ctx = _box_of_blocks(shape)
    nb = len(ctx.active_blocks())
    rng = np.random.default_rng(nb)
    r = rng.normal(size=(nb, 512))
    if nb > 27:
        r[: nb // 3] = 0.0  # blocks whose whole window holds no residual are skipped
    r = _t(r.ravel())
    ctx.set_learned_preconditioner(_t(U.init_params(9) + 0.01 * rng.normal(size=U.param_count())))
    z, ref = torch.zeros(nb * 512, device="cuda"), torch.zeros(nb * 512, device="cuda")
    ctx.apply_learned(r, z, kernels=0)
    ctx.apply_learned(r, ref, kernels=1)
    z, ref = z.cpu().numpy(), ref.cpu().numpy()
    assert np.any(ref != 0.0)
    assert _rel(z, ref) <= 3e-2
    ctx.close()


@pytest.mark.parametrize("shape", [(4, 4, 5), (8, 10, 2), (11, 9, 10)])
def test_tensor_core_inference_with_several_blocks_per_cta(shape):
    """The inference where a CTA of the convolutions takes block after block through its two operand and
    two accumulator stages: 150 and 297 blocks, one or two more than one CTA per SM and two, and 1320,
    four and more for each of two CTAs per SM. The residual is zero in parts of the box, so that
    blocks to skip lie between others in a CTA's sequence. Against the FP32 forward, each
    block for itself: 3e-2 of its largest value, as the tests above for all of them."""
    import torch

    ctx = _box_of_blocks(shape)
    blocks = ctx.active_blocks()
    nb = len(blocks)
    rng = np.random.default_rng(nb)
    r = rng.normal(size=(nb, 512))
    if nb > 1000:  # cubes of 4^3 blocks all over the box
        r[(blocks // 4).sum(1) % 2 == 1] = 0.0
    else:
        r[blocks[:, 0] < len(np.unique(blocks[:, 0])) // 2] = 0.0
    near = {tuple(b + d) for b in blocks[np.any(r != 0.0, 1)] for d in np.indices((3, 3, 3)).reshape(3, -1).T - 1}
    idle = np.array([tuple(b) not in near for b in blocks])
    assert 0 < idle.sum() < nb // 2
    r = _t(r.ravel())
    ctx.set_learned_preconditioner(_t(U.init_params(9) + 0.01 * rng.normal(size=U.param_count())))
    z, ref = torch.full((nb * 512,), 5.0, device="cuda"), torch.full((nb * 512,), 5.0, device="cuda")
    ctx.apply_learned(r, z, kernels=0)
    ctx.apply_learned(r, ref, kernels=1)
    z, ref = z.cpu().numpy().reshape(nb, 512), ref.cpu().numpy().reshape(nb, 512)
    assert np.all(z[idle] == 0.0) and np.all(ref[idle] == 0.0)
    assert np.all(np.abs(z - ref).max(1) <= 3e-2 * np.abs(ref).max(1))
    ctx.close()


@pytest.mark.parametrize("tensor_cores", [False, True])
def test_training_passes_in_a_row_are_ordered(tensor_cores):
    """Kernels of a pass may be scheduled before their predecessors end, and each waits before it reads:
    Adam, forward and backward issued in a row give the bits that the same calls give with the device
    idle before each."""
    import torch

    rng = np.random.default_rng(15)
    x, gy = _t(rng.normal(size=(45, 2, 10, 10, 10))), _t(rng.normal(size=(45, 512)))
    th = _t(U.init_params(2) + 0.01 * rng.normal(size=U.param_count()))
    unet = fb.UNet(45, tensor_cores=tensor_cores)
    results = []
    for idle in (True, False, False):
        p, m, v = th.clone(), torch.zeros_like(th), torch.zeros_like(th)
        y, g = torch.zeros((45, 512), device="cuda"), torch.zeros_like(th)
        for step in range(1, 13):
            for call in (lambda: unet.forward(p, x, y), lambda: unet.backward(p, gy, g),
                         lambda: fb.UNet.adam_step(p, g, m, v, step)):
                call()
                if idle:
                    torch.cuda.synchronize()
        results.append(torch.cat([p, g, y.ravel()]).cpu().numpy())
    for r in results[1:]:
        np.testing.assert_array_equal(r, results[0])
    unet.close()


@pytest.mark.parametrize("tensor_cores", [False, True])
def test_weight_gradients_end_before_the_stream_goes_on(tensor_cores):
    """The weight gradients run beside the data gradients on a stream of the handle's own: what the
    caller's stream does right after the backward (overwriting its inputs, another forward into the same
    activations) does not reach them. The same bits as with the device idle in between."""
    import torch

    rng = np.random.default_rng(17)
    x, gy = _t(rng.normal(size=(40, 2, 10, 10, 10))), _t(rng.normal(size=(40, 512)))
    th = _t(U.init_params(4) + 0.01 * rng.normal(size=U.param_count()))
    unet = fb.UNet(40, tensor_cores=tensor_cores)
    stream = torch.cuda.Stream()
    grads = []
    torch.cuda.synchronize()
    for idle in (True, False, False):
        with torch.cuda.stream(stream):
            p, up, y, g = th.clone(), gy.clone(), torch.zeros((40, 512), device="cuda"), torch.zeros_like(th)
            unet.forward(p, x, y, stream=stream.cuda_stream)
            unet.backward(p, up, g, stream=stream.cuda_stream)
            if idle:
                torch.cuda.synchronize()
            out = g.clone()
            p.zero_()
            up.fill_(float("nan"))
            unet.forward(p, x, y, stream=stream.cuda_stream)
        torch.cuda.synchronize()
        grads.append(out.cpu().numpy())
    assert np.all(np.isfinite(grads[0])) and np.any(grads[0] != 0.0)
    for g in grads[1:]:
        np.testing.assert_array_equal(g, grads[0])
    unet.close()


FIRST_CALLS = """
import threading
import torch
import fluidity_b200 as fb

threads, tensor_cores = 6, {tensor_cores}
torch.manual_seed(1)
x = torch.randn((8, 2, 10, 10, 10), device="cuda")
x[:, 1] = 1.0
p = 0.1 * torch.randn(fb.UNet.param_count(), device="cuda")
torch.cuda.synchronize()
start, results = threading.Barrier(threads), [None] * threads


def work(k):
    net = fb.UNet(8, tensor_cores=tensor_cores)
    y, g, gy, loss = torch.zeros((8, 512), device="cuda"), torch.zeros_like(p), torch.zeros((8, 512), device="cuda"), torch.zeros(1, device="cuda")
    torch.cuda.synchronize()
    start.wait()
    net.forward(p, x, y)
    fb.UNet.block_residual_loss(y, x, loss, gy)
    net.backward(p, gy, g)
    torch.cuda.synchronize()
    results[k] = torch.cat([y.ravel(), g, loss])
    net.close()


ts = [threading.Thread(target=work, args=(k,)) for k in range(threads)]
[t.start() for t in ts]
[t.join() for t in ts]
assert all(r is not None and bool(torch.isfinite(r).all()) for r in results), [r is None for r in results]
assert all(torch.equal(r, results[0]) for r in results)
"""


@pytest.mark.parametrize("tensor_cores", [False, True])
def test_first_calls_of_several_threads(tensor_cores):
    """Threads with a handle each whose first passes start together, in a process of their own so that
    no kernel's shared-memory attribute is set yet: no launch precedes it, and all get the same bits."""
    import subprocess
    import sys
    from pathlib import Path

    root = Path(__file__).resolve().parent.parent
    r = subprocess.run([sys.executable, "-c", FIRST_CALLS.format(tensor_cores=tensor_cores)], cwd=root, timeout=300,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]


def test_network_on_a_second_device():
    """Kernel attributes belong to a device: after a pass on one GPU the same pass runs on another."""
    import torch

    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    rng, results = np.random.default_rng(3), []
    x, gy, th = rng.normal(size=(4, 2, 10, 10, 10)), rng.normal(size=(4, 512)), U.init_params(2)
    for device in (0, 1):
        with torch.cuda.device(device):
            net, P, X, DY = fb.UNet(4), _t(th), _t(x), _t(gy)
            Y, G = torch.zeros((4, 512), device="cuda"), torch.zeros_like(P)
            net.forward(P, X, Y)
            net.backward(P, DY, G)
            torch.cuda.synchronize()
            results.append(torch.cat([Y.ravel(), G]).cpu().numpy())
            net.close()
    np.testing.assert_array_equal(results[0], results[1])

"""Which inputs the reverse mode's one-launch forms take.  Their kernels read and
write float32 (n, 3) arrays on the plan's device and check nothing, so any other
input has to go through torch's own rules (broadcasting, promotion, its errors)
in the tensor form.  No GPU: the launch is replaced by a failure."""
import types

import pytest

torch = pytest.importorskip("torch")

N = 5
BOX = torch.tensor([2.0, 3.0, 4.0])


def _model(device="cpu"):
    md = types.SimpleNamespace(n=N, mass=2.0, dt=0.01, respa=3,
                               r=torch.zeros(N, 3, device=device))
    return types.SimpleNamespace(md=md, fused_inner=True, box_f=BOX, thermo=None)


@pytest.fixture
def stubs(monkeypatch):
    from hymd_gb300 import reverse

    def refuse(*a):
        raise AssertionError("the kernel form took this input")

    monkeypatch.setattr(reverse._InnerLoop, "apply", refuse)
    monkeypatch.setattr(reverse, "bonded_force", lambda x, model: -0.5 * x)
    monkeypatch.setattr(reverse, "field_force", lambda x, chi, model: torch.sin(x))
    return reverse


def _by_hand(x, v, fs, fb, model):
    m, dt, n_in = model.md.mass, model.md.dt, model.md.respa
    v = v + (0.5 * n_in * dt / m) * fs
    for _ in range(n_in):
        v = v + (0.5 * dt / m) * fb
        x = torch.remainder(x + dt * v, model.box_f)
        fb = -0.5 * x
        v = v + (0.5 * dt / m) * fb
    fs = torch.sin(x)
    return x, v + (0.5 * n_in * dt / m) * fs, fs, fb


@pytest.mark.parametrize("shape", [(1, 3), (3,), (N, 1), (N, 3)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16, torch.float64])
def test_inner_loop_other_inputs(stubs, shape, dtype):
    g = torch.Generator().manual_seed(3)
    x = torch.rand(N, 3, generator=g) + 0.5
    v = torch.randn(shape, generator=g).to(dtype)
    fs, fb = torch.sin(x), -0.5 * x
    model = _model()
    got = stubs.respa_step(x, v, fs, fb, None, model)
    for a, b in zip(got, _by_hand(x, v, fs, fb, model)):
        assert torch.equal(a, b)


def test_inner_loop_rule(stubs):
    """The rule itself, on tensors that say they are on a GPU (meta tensors have
    no memory: only what the rule reads is there)."""
    class Cuda:
        def __init__(self, shape=(N, 3), dtype=torch.float32, device="cuda:0", is_cuda=True):
            self.shape, self.dtype, self.is_cuda = torch.Size(shape), dtype, is_cuda
            self.device = torch.device(device)

    model = _model()
    model.md.r = Cuda()
    ok = lambda *t: stubs._inner_fusable(*t, model)  # noqa: E731
    good = Cuda()
    assert ok(good, good, good, good)
    for bad in (Cuda((1, 3)), Cuda((3,)), Cuda((N, 1)), Cuda((N + 1, 3)), Cuda((N, 3, 1)),
                Cuda(dtype=torch.bfloat16), Cuda(dtype=torch.float64), Cuda(device="cuda:1"),
                Cuda(device="cpu", is_cuda=False)):
        for k in range(4):
            args = [good] * 4
            args[k] = bad
            assert not ok(*args)
    model.fused_inner = False
    assert not ok(good, good, good, good)


@pytest.mark.gpu
def test_one_velocity_for_all_beads():
    """A (1, 3) start velocity broadcasts, and gets a gradient of its own shape: the
    first step runs step by step, the second in the kernels.  Against the same
    velocity written out, whose first step is the kernels': FP32 in another order
    over two steps, 1e-4 of the loss and 1e-3 of the gradients (that sum over beads
    of both signs)."""
    from hymd_gb300 import systems
    from hymd_gb300.hamiltonian import get_hamiltonian
    from hymd_gb300.md import RespaMD
    from hymd_gb300.reverse import ForceModel, profile_loss
    s = systems.homopolymer_melt(seed=4, n_chains=33, length=10, box=5.6, mesh=16)
    cfg = s["config"]
    cfg.barostat, cfg.respa_inner, cfg.time_step = None, 3, 0.01
    md = RespaMD(s["positions"], s["velocities"], s["types"], cfg, get_hamiltonian(cfg),
                 topology=s["topology"])
    model = ForceModel(md)
    chi = torch.tensor([[0.0, 5.0], [5.0, 0.0]], dtype=torch.float64, device="cuda")
    target = torch.zeros(2, 20, device="cuda")
    out = []
    for rows in (1, md.n):
        v0 = torch.tensor([[0.3, -0.2, 0.5]], device="cuda").expand(rows, 3).clone()
        v0.requires_grad_(True)
        loss, _ = profile_loss(md.r.clone(), v0, chi, model, 2, target, n_bins=20)
        (g,) = torch.autograd.grad(loss, v0)
        assert g.shape == (rows, 3)
        out.append((float(loss.detach()), g.double().sum(0), g.double().abs().sum(0)))
    md.check_errors()
    assert abs(out[0][0] - out[1][0]) <= 1e-4 * out[1][0]
    assert bool(((out[0][1] - out[1][1]).abs() <= 1e-3 * out[1][2]).all())


@pytest.fixture
def profile_stub(monkeypatch):
    from hymd_gb300 import reverse

    def refuse(*a):
        raise AssertionError("the kernel form took this input")

    monkeypatch.setattr(reverse._ZProfile, "apply", refuse)
    return reverse


class _Claims(torch.Tensor):
    """A CPU tensor that says it is on a GPU."""
    is_cuda = True


def _claims(t):
    return t.as_subclass(_Claims)


@pytest.mark.parametrize("types", [torch.zeros(N - 1, dtype=torch.int32),
                                   torch.zeros(1, dtype=torch.int32),
                                   torch.zeros((), dtype=torch.int32),
                                   torch.zeros(N + 2, dtype=torch.int32)])
def test_profile_types_of_another_length(profile_stub, types):
    x = torch.rand(N, 3)
    a, b = _claims(x), _claims(types)
    if types.numel() == 1:  # one species: broadcasts
        want = profile_stub._z_profile_torch(x, types, 1, 4, [1.0, 1.0, 1.0])
        assert torch.equal(profile_stub.z_profile(a, b, 1, 4, [1.0, 1.0, 1.0]), want)
    else:
        with pytest.raises((RuntimeError, IndexError)):
            profile_stub.z_profile(a, b, 1, 4, [1.0, 1.0, 1.0])


def test_profile_box_gradient(profile_stub):
    x, t = torch.rand(N, 3), torch.zeros(N, dtype=torch.int32)
    box = torch.tensor([1.0, 1.0, 1.0], requires_grad=True)
    p = profile_stub.z_profile(_claims(x), _claims(t), 1, 4, box)
    (g,) = torch.autograd.grad(p.sum(), box)
    assert float(g.abs().sum()) > 0


def test_profile_transforms(profile_stub, monkeypatch):
    """vmap, torch.func.grad, forward mode and tracing take the tensor form."""
    import torch.autograd.forward_ad as fwd
    from torch.fx.experimental.proxy_tensor import make_fx
    x, t = torch.rand(N, 3) + 0.01, torch.zeros(N, dtype=torch.int32)
    seen = []

    def rule(x, types, *a):  # as on a GPU: where the tensors live left out
        seen.append(profile_stub._untransformed(x, types))
        return seen[-1]

    monkeypatch.setattr(profile_stub, "_profile_fusable", rule)
    f = lambda y: profile_stub.z_profile(y, t, 1, 4, [2.0] * 3)  # noqa: E731
    plain = lambda y: profile_stub._z_profile_torch(y, t, 1, 4, [2.0] * 3)  # noqa: E731
    xs, w = torch.stack([x, x + 0.1]), torch.arange(4.0)
    assert torch.allclose(torch.vmap(f)(xs), torch.stack([plain(xs[0]), plain(xs[1])]))
    assert torch.allclose(torch.func.grad(lambda y: (f(y) * w).sum())(x),
                          torch.func.grad(lambda y: (plain(y) * w).sum())(x))
    with fwd.dual_level():
        d = fwd.make_dual(x, torch.ones_like(x))
        assert fwd.unpack_dual(f(d)).tangent is not None
    torch.jit.trace(f, x, check_trace=False)
    make_fx(f)(x)
    assert len(seen) >= 5 and not any(seen)
    assert profile_stub._untransformed(x, t)


def test_profile_rule(profile_stub):
    x, t = torch.rand(N, 3), torch.zeros(N, dtype=torch.int32)

    class Cuda:
        """What the rule reads of a plain tensor on a GPU."""
        def __init__(self, base, device="cuda:0", is_cuda=True, contiguous=True):
            self.dtype, self.shape, self.is_cuda = base.dtype, base.shape, is_cuda
            self.device, self._c = torch.device(device), contiguous

        def dim(self):
            return len(self.shape)

        def is_contiguous(self):
            return self._c

    with pytest.MonkeyPatch.context() as mp:
        mp.setattr(profile_stub, "_untransformed", lambda *a: True)
        ok = profile_stub._profile_fusable
        box = [1.0, 2.0, 3.0]
        assert ok(Cuda(x), Cuda(t), 2, 10, box)
        assert not ok(Cuda(x), Cuda(t[:-1]), 2, 10, box)
        assert not ok(Cuda(x), Cuda(t[:1]), 2, 10, box)
        assert not ok(Cuda(x), Cuda(t.reshape(N, 1)), 2, 10, box)
        assert not ok(Cuda(x), Cuda(t, device="cuda:1"), 2, 10, box)
        assert not ok(Cuda(x), Cuda(t, device="cpu", is_cuda=False), 2, 10, box)
        assert not ok(Cuda(x), Cuda(t.long()), 2, 10, box)
        assert not ok(Cuda(x), Cuda(t, contiguous=False), 2, 10, box)
        assert not ok(Cuda(x, contiguous=False), Cuda(t), 2, 10, box)
        assert not ok(Cuda(x.double()), Cuda(t), 2, 10, box)
        assert not ok(Cuda(x[:, :2]), Cuda(t), 2, 10, box)
        assert not ok(Cuda(x[:0]), Cuda(t[:0]), 2, 10, box)
        assert not ok(Cuda(x), Cuda(t), 0, 10, box)
        assert not ok(Cuda(x), Cuda(t), 2, 0, box)
        assert not ok(Cuda(x), Cuda(t), 2, 2 ** 28, box)
        assert not ok(Cuda(x), Cuda(t), 2, 10, torch.tensor(box))
        assert not ok(Cuda(x), Cuda(t), 2, 10, [1.0, torch.tensor(2.0), 3.0])
        assert not ok(Cuda(x), Cuda(t), 2, 10, [1.0, 2.0, 0.0])
        assert not ok(Cuda(x), Cuda(t), 2, 10, [1.0, -2.0, 3.0])
        assert not ok(Cuda(x), Cuda(t), 2, 10, [1.0, 2.0, float("nan")])
    assert not profile_stub._untransformed(_claims(x), t)


@pytest.mark.gpu
def test_profile_second_derivative():
    """Derivatives of the gradient with respect to the incoming one, and a forward-mode
    derivative, against the tensor form in 64 bits.  A bead's weight is linear in its z
    (slope n_bins / Lz), so both are sums of at most n such terms, exact to FP32
    rounding: 1e-5 of their largest."""
    import torch.autograd.forward_ad as fwd
    from hymd_gb300.reverse import _z_profile_torch, z_profile
    gen = torch.Generator(device="cuda").manual_seed(2)
    n, T, bins, box = 1000, 2, 10, [3.0, 4.0, 5.0]
    x = torch.rand(n, 3, generator=gen, device="cuda") * 2.9
    types = (torch.arange(n, device="cuda") % T).int()
    g, u = torch.randn(T, bins, generator=gen, device="cuda"), torch.rand_like(x)
    out = []
    for form, y, h, w in ((z_profile, x, g, u), (_z_profile_torch, x.double(), g.double(),
                                                 u.double())):
        y, h = y.clone().requires_grad_(True), h.clone().requires_grad_(True)
        (g1,) = torch.autograd.grad(form(y, types, T, bins, box), y, h, create_graph=True)
        (g2,) = torch.autograd.grad((g1 * w).sum(), h)
        with fwd.dual_level():
            t = fwd.unpack_dual(form(fwd.make_dual(y.detach(), w), types, T, bins, box)).tangent
        out.append((g2, t))
    for a, b in zip(*out):
        assert float((a.double() - b).abs().max()) <= 1e-5 * float(b.abs().max())
    # one species for all beads
    one = torch.zeros(1, dtype=torch.int32, device="cuda")
    p = z_profile(x, one, 1, bins, box)
    want = z_profile(x, one.expand(n).contiguous(), 1, bins, box)
    assert float((p - want).abs().max()) <= 1e-5 * float(want.max())


def test_profile_on_another_device(monkeypatch):
    """The kernels are launched on the current device: tensors of another one take the
    tensor form, which follows them there."""
    from hymd_gb300 import reverse

    class Cuda(torch.Tensor):
        is_cuda = True
        device = torch.device("cuda", 1)

    x = torch.rand(N, 3).as_subclass(Cuda)
    t = torch.zeros(N, dtype=torch.int32).as_subclass(Cuda)
    monkeypatch.setattr(reverse, "_plain", lambda *a: True)
    for current, want in ((0, False), (1, True)):
        monkeypatch.setattr(torch.cuda, "current_device", lambda: current)
        assert reverse._untransformed(x, t) is want

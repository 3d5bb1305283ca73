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

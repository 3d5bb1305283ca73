"""Scratch that is set up on first use is ready for that use on any stream: the first
FP64 energy, charge chain and GPE solve of a context on a side stream, with the
default stream busy, give the bits of an idle default stream.  Under capture the first
energy is refused, and the context stays usable."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

T, N = 2, 3000


def _pm():
    from hymd_gb300 import _lib
    from hymd_gb300.field import ParticleMesh
    pm = ParticleMesh([24] * 3, [6.0] * 3, T)
    _lib.call("hpf_ctx_set_functional", pm._h, _lib.dvec([2.0, 1.5, 1.5, 2.0]),
              _lib.dvec([-1.0] * T), 0.5, 0.4)
    return pm


def _inputs():
    rng = np.random.default_rng(8)
    r = torch.as_tensor((rng.uniform(0, 0.999, (N, 3)) * 6).astype(np.float32), device="cuda")
    types = (torch.arange(N, device="cuda") % T).int()
    q = torch.as_tensor(rng.choice([-1.0, 0.0, 1.0], N).astype(np.float32), device="cuda")
    idx = torch.nonzero(q != 0).reshape(-1).to(torch.int32).contiguous()
    return r, types, q, idx


def _energy(pm, r, types, q, idx):
    from hymd_gb300 import _lib
    out = torch.zeros(32, dtype=torch.float64, device="cuda")
    _lib.call("hpf_energy_fp64", pm._h, _lib.ptr(r), _lib.ptr(types), N, _lib.dvec([1.0] * T),
              _lib.ptr(q), _lib.dvec([0.3, -0.2]), 1.7, _lib.ptr(out), _lib.stream_ptr())
    return [out]


def _chains(pm, r, types, q, idx):
    from hymd_gb300 import _lib
    F, E = torch.zeros_like(r), torch.zeros_like(r)
    s, e = (torch.zeros(8, dtype=torch.float64, device="cuda") for _ in range(2))
    _lib.call("hpf_field_pic_step", pm._h, _lib.ptr(r), _lib.ptr(types), N, _lib.dvec([1.0] * T),
              _lib.ptr(F), _lib.ptr(s), None, _lib.ptr(q), _lib.ptr(idx), idx.numel(), 1.7,
              _lib.ptr(E), _lib.ptr(e), None, 0, _lib.stream_ptr())
    return [F, E, s, e]


@pytest.mark.parametrize("what", [_energy, _chains])
def test_first_use_on_a_side_stream(what):
    args = _inputs()
    want = what(_pm(), *args)
    torch.cuda.synchronize()
    pm = _pm()
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    torch.cuda._sleep(20_000_000)  # the default stream is busy for about 10 ms
    with torch.cuda.stream(s):
        s_args = args
        got = what(pm, *s_args)
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    pm.check_errors()


def test_first_energy_under_capture_is_refused():
    from hymd_gb300 import _lib
    args = _inputs()
    want = _energy(_pm(), *args)[0]
    pm = _pm()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        with pytest.raises(_lib.HPFError):
            _energy(pm, *args)
    torch.cuda.synchronize()
    got = _energy(pm, *args)[0]
    assert torch.equal(got, want)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = _energy(pm, *args)[0]
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)

"""The mesh context's functional on a side stream that is still busy: each force
evaluation uses the functional set before it, whether it was formed on the device
from chi (queued) or came from the host (copied), in either order.  The same calls
on an idle default stream give the same bits."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

T, N = 2, 3000


def _system():
    from hymd_gb300.field import ParticleMesh
    rng = np.random.default_rng(6)
    pm = ParticleMesh([24] * 3, [6.0] * 3, T)
    r = torch.as_tensor((rng.uniform(0, 0.999, (N, 3)) * 6).astype(np.float32), device="cuda")
    types = (torch.arange(N, device="cuda") % T).int()
    return pm, r, types


def _force(pm, r, types):
    from hymd_gb300 import _lib
    F = torch.zeros_like(r)
    _lib.call("hpf_field_step", pm._h, _lib.ptr(r), _lib.ptr(types), N, _lib.dvec([1.0] * T),
              _lib.ptr(F), None, None, None, _lib.stream_ptr())
    return F


def _calls(pm, r, types, chis, order):
    """Forces under chis[0..] set alternately from the device and the host."""
    from hymd_gb300 import _lib
    from hymd_gb300.adjoint import _set, functional_coefficients
    out = []
    for k, chi in enumerate(chis):
        if (k + order) % 2 == 0:
            _lib.call("hpf_ctx_set_functional_chi", pm._h, _lib.ptr(chi), 1, 1, 0.05, 8.3, 8.1,
                      0.5, _lib.stream_ptr())
        else:
            Q, b, c = functional_coefficients("DefaultWithChi", HOST[k], 0.05, 8.3, 8.1)
            _set(pm, Q, b, c, 0.5)
        out.append(_force(pm, r, types))
    return out


HOST = [np.array([[0.0, x], [x, 0.0]]) for x in (5.0, 40.0, -10.0, 20.0)]


@pytest.mark.parametrize("order", [0, 1])
def test_side_stream(order):
    pm, r, types = _system()
    chis = [torch.as_tensor(h, device="cuda") for h in HOST]
    want = _calls(pm, r, types, chis, order)
    torch.cuda.synchronize()
    assert not torch.equal(want[0], want[1])
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        torch.cuda._sleep(20_000_000)  # about 10 ms: what follows is queued behind it
        got = _calls(pm, r, types, chis, order)
    s.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    pm.check_errors()


def test_host_setter_without_a_stream():
    """hpf_ctx_set_functional waits for a functional queued on another stream."""
    from hymd_gb300 import _lib
    from hymd_gb300.adjoint import functional_coefficients
    pm, r, types = _system()
    chi = torch.as_tensor(HOST[0], device="cuda")
    Q, b, c = functional_coefficients("DefaultWithChi", HOST[1], 0.05, 8.3, 8.1)
    q, bb = _lib.dvec(Q.reshape(-1)), _lib.dvec(b)
    _lib.call("hpf_ctx_set_functional", pm._h, q, bb, float(c), 0.5)
    want = _force(pm, r, types)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        torch.cuda._sleep(20_000_000)
        _lib.call("hpf_ctx_set_functional_chi", pm._h, _lib.ptr(chi), 1, 1, 0.05, 8.3, 8.1, 0.5,
                  _lib.stream_ptr())
    _lib.call("hpf_ctx_set_functional", pm._h, q, bb, float(c), 0.5)
    got = _force(pm, r, types)
    torch.cuda.synchronize()
    assert torch.equal(got, want)

"""HpfKick.defer took the place of padding that a C caller never had to set: only 1
defers the velocity sums, any other content gives the factors in the same call, with the
same bits."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_any_other_padding_does_not_defer():
    from hymd_gb300 import _lib
    from hymd_gb300.field import ParticleMesh
    rng = np.random.default_rng(7)
    n = 1000
    r = torch.as_tensor((rng.uniform(0, 0.999, (n, 3)) * 8).astype(np.float32), device="cuda")
    types = torch.zeros(n, dtype=torch.int32, device="cuda")
    v0 = torch.as_tensor(rng.normal(0, 0.2, (n, 3)).astype(np.float32), device="cuda")
    table = torch.as_tensor(np.array([0.3, 3.0 * n] * 4), device="cuda")
    pm = ParticleMesh([16, 16, 16], [8.0] * 3, 1)
    _lib.call("hpf_ctx_set_functional", pm._h, _lib.dvec([2.0]), _lib.dvec([-1.0]), 0.0, 0.5)
    a = _lib.CsvrArgs()
    a.n_groups, a.remove_com, a.n_steps, a.stride, a.advance, a.every = 1, 1, 4, 2, 1, 1
    a.count[0] = float(n)
    a.mass, a.gas_constant, a.target_temperature, a.c = 72.0, 0.0083144621, 323.0, 0.05
    out = []
    for padding in (0, 2, -1, 0x7ffd1234):
        v, force = v0.clone(), torch.zeros_like(v0)
        state = torch.zeros(16, dtype=torch.float64, device="cuda")
        counter = torch.ones(4, dtype=torch.int32, device="cuda")
        ws = _lib.new_workspace()
        k = _lib.Kick()
        k.v, k.mass, k.dt_outer, k.defer = v.data_ptr(), 72.0, 0.3, padding
        k.thermo = _lib.ctypes.pointer(a)
        k.randoms, k.counter, k.state = table.data_ptr(), counter.data_ptr(), state.data_ptr()
        k.ws = ws.data_ptr()
        _lib.call("hpf_field_step", pm._h, _lib.ptr(r), _lib.ptr(types), n, _lib.dvec([1.0]),
                  _lib.ptr(force), None, None, _lib.ctypes.byref(k), _lib.stream_ptr())
        assert int(counter[0]) == 2
        out.append((v, state))
    for v, state in out[1:]:
        assert torch.equal(v, out[0][0]) and torch.equal(state, out[0][1])
    pm.check_errors()

"""The thermostat formed and applied in one launch from the readout's block
partials (HpfKick.defer, hpf_csvr_apply) against the readout's own reduction
followed by hpf_csvr_scale: one and two coupling groups, with and without COM
removal, velocities off a 16-byte boundary, a last float4 that is not full,
and bead counts around the grid's blocks.

Both sum the same per-thread FP32 partials in double-float arithmetic, in
another order: the sums agree to about 1e-13 and the float32 scale factors to
one rounding, so velocities within 2 ulp (2.4e-7 relative to their RMS size)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,groups,com,offset", [
    (1, 1, True, 0), (85, 1, True, 0), (257, 2, True, 0), (1021, 1, False, 0),
    (4097, 1, True, 1), (90001, 2, False, 0), (250003, 1, True, 0)])
def test_apply_matches_scale(n, groups, com, offset):
    from hymd_gb300 import _lib
    from hymd_gb300.field import ParticleMesh
    rng = np.random.default_rng(n)
    box = np.array([8.0, 8.0, 8.0])
    r = torch.as_tensor(np.mod(rng.uniform(0, 8, (n, 3)), 8).astype(np.float32), device="cuda")
    types = torch.zeros(n, dtype=torch.int32, device="cuda")
    v0 = torch.as_tensor(rng.normal(0, 0.2, (n, 3)).astype(np.float32), device="cuda")
    grp = torch.as_tensor((np.arange(n) % groups).astype(np.int32), device="cuda")
    table = torch.as_tensor(np.array([0.3, 3.0 * n, -0.7, 2.5 * n] * 4), device="cuda")
    pm = ParticleMesh([16, 16, 16], box, 1)
    _lib.call("hpf_ctx_set_functional", pm._h, _lib.dvec([2.0]), _lib.dvec([-1.0]), 0.0, 0.5)
    a = _lib.CsvrArgs()
    a.n_groups, a.remove_com, a.n_steps, a.stride = groups, int(com), 4, 4
    a.offset, a.advance, a.every = 0, 1, 1
    counts = np.bincount(np.arange(n) % groups, minlength=2)
    a.count[0], a.count[1] = float(counts[0]), float(counts[1])
    a.mass, a.gas_constant, a.target_temperature, a.c = 72.0, 0.0083144621, 323.0, 0.05
    out = []
    for defer in (0, 1):
        buf = torch.zeros(3 * n + 4, dtype=torch.float32, device="cuda")
        v = buf[offset:offset + 3 * n].view(n, 3)
        v.copy_(v0)
        force = torch.zeros((n, 3), dtype=torch.float32, device="cuda")
        state = torch.zeros(16, dtype=torch.float64, device="cuda")
        counter = torch.ones(4, dtype=torch.int32, device="cuda")
        err = torch.zeros(8, dtype=torch.int32, device="cuda")
        ws = _lib.new_workspace()
        k = _lib.Kick()
        k.v, k.mass, k.dt_outer, k.defer = v.data_ptr(), 72.0, 0.3, defer
        k.thermo = _lib.ctypes.pointer(a)
        k.group = grp.data_ptr() if groups > 1 else None
        k.randoms, k.counter, k.state = table.data_ptr(), counter.data_ptr(), state.data_ptr()
        k.ws, k.d_err = ws.data_ptr(), err.data_ptr()
        g = grp if groups > 1 else None
        for _ in range(2):
            _lib.call("hpf_field_step", pm._h, _lib.ptr(r), _lib.ptr(types), n, _lib.dvec([1.0]),
                      _lib.ptr(force), None, None, _lib.ctypes.byref(k), _lib.stream_ptr())
            if defer:
                _lib.call("hpf_csvr_apply", _lib.ptr(v), _lib.ptr(g), n, _lib.ctypes.byref(a),
                          _lib.ptr(table), _lib.ptr(counter), _lib.ptr(state), _lib.ptr(ws),
                          _lib.ptr(err), _lib.stream_ptr())
            else:
                _lib.call("hpf_csvr_scale", _lib.ptr(v), _lib.ptr(g), n, _lib.ptr(state),
                          int(com), _lib.stream_ptr())
        torch.cuda.synchronize()
        assert int(err[0]) == 0 and int(counter[0]) == 3
        out.append((v.double().cpu(), state.cpu(), float(buf[3 * n + offset:].abs().sum())))
    (va, sa, ta), (vb, sb, tb) = out
    rms = float(va.square().mean().sqrt())
    assert float((va - vb).abs().max()) <= 2.4e-7 * max(rms, float(va.abs().max()))
    assert torch.allclose(sa, sb, rtol=1e-6, atol=1e-9)
    assert ta == 0.0 and tb == 0.0  # nothing written past the velocities

"""Field forces with k-space tiles that transform v in place (tiles too large
for a block of their own for it) against the 4-column tile, which does not:
the same arithmetic per column, so the same bits; lengths 2^a and 3 * 2^a,
columns per round that do and do not divide the tile."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh,T,wide", [((128, 16, 16), 3, 16), ((256, 16, 16), 3, 8),
                                         ((192, 24, 24), 3, 8), ((96, 48, 48), 4, 16),
                                         ((128, 16, 32), 5, 8), ((64, 16, 16), 6, 16)])
def test_widths_agree(mesh, T, wide):
    from hymd_gb300 import _lib
    from hymd_gb300.field import ParticleMesh
    rng = np.random.default_rng(T)
    n = 6007
    box = 0.4 * np.array(mesh)
    pm = ParticleMesh(mesh, box, T)
    A = rng.normal(size=(T, T))
    _lib.call("hpf_ctx_set_functional", pm._h, _lib.dvec((A @ A.T).reshape(-1)),
              _lib.dvec([-1.0] * T), 0.0, 0.5)
    r = torch.as_tensor((rng.uniform(0, 0.999, (n, 3)) * box).astype(np.float32), device="cuda")
    types = torch.as_tensor(rng.integers(0, T, n).astype(np.int32), device="cuda")
    assert wide in pm.spectral_tiles_allowed
    out = []
    for w in (4, wide):
        pm.spectral_tile = w
        F = torch.zeros_like(r)
        sums = torch.zeros(8, dtype=torch.float64, device="cuda")
        _lib.call("hpf_field_step", pm._h, _lib.ptr(r), _lib.ptr(types), n, _lib.dvec([1.0] * T),
                  _lib.ptr(F), _lib.ptr(sums), None, None, _lib.stream_ptr())
        out.append((F, sums))
    pm.check_errors()
    assert torch.equal(out[0][0], out[1][0])
    assert torch.allclose(out[0][1][:4], out[1][1][:4], rtol=1e-6)

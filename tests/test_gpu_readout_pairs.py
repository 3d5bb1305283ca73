"""The readout's paired loads (even n2, 8-byte aligned mesh) against its single
loads, taken for the same mesh 4 bytes off: the same values in the same order,
so the same bits; beads in first and last cells of each axis, n2 = 2."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh,T", [((4, 4, 2), 1), ((5, 7, 6), 2), ((16, 9, 16), 3),
                                    ((24, 24, 24), 2)])
def test_pairs_match_singles(mesh, T):
    from hymd_gb300 import _lib
    from hymd_gb300.field import ParticleMesh
    rng = np.random.default_rng(mesh[2])
    n = 3001
    box = 0.4 * np.array(mesh)
    r = (rng.uniform(0, 0.9999, (n, 3)) * box).astype(np.float32)
    r[:64, 2] = np.float32(box[2]) * np.linspace(0.97, 0.9999, 64, dtype=np.float32)
    r[64:128, 2] = 0.0
    R = torch.as_tensor(r, device="cuda")
    types = torch.as_tensor(rng.integers(0, T, n).astype(np.int32), device="cuda")
    pm = ParticleMesh(mesh, box, T)
    m = 3 * T * pm.M
    buf = torch.randn(m + 4, device="cuda")
    off = torch.empty(m + 4, device="cuda")
    off[1:m + 1] = buf[:m]
    out = []
    for mesh_t in (buf[:m], off[1:m + 1]):
        F = torch.zeros(n, 3, device="cuda")
        _lib.call("hpf_readout", pm._h, _lib.ptr(mesh_t), _lib.ptr(R), _lib.ptr(types), n,
                  _lib.ptr(F), _lib.stream_ptr())
        out.append(F)
    pm.check_errors()
    assert torch.equal(out[0], out[1]) and float(out[0].abs().max()) > 0

"""FP64 energy sums in double-float arithmetic (the fused meshes) against the
cuFFT D2Z path on the same deposits: every pair of transform lengths at its
smallest, largest and 3 * 2^a sizes, one to eight types, with and without
charges, two calls in a row (the accumulators are left clear).

Both start from the same integers; the transforms carry 48 and 53 bits, so
the sums of up to 10^6 terms agree to about 1e-13: 1e-11 of each sum's scale
(the cross sums C cancel, so their scale is that of the type densities')."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh,T,q", [
    ((8, 16, 16), 1, True), ((16, 16, 32), 2, False), ((32, 64, 16), 3, True),
    ((64, 32, 64), 8, True), ((24, 24, 24), 2, True), ((48, 48, 48), 4, False),
    ((192, 24, 24), 1, True), ((96, 96, 96), 2, True), ((256, 16, 128), 3, False),
    ((16, 128, 128), 5, True), ((128, 128, 64), 1, False)])
def test_matches_d2z(mesh, T, q):
    from hymd_gb300 import _lib
    from hymd_gb300.field import ParticleMesh
    rng = np.random.default_rng(sum(mesh) + T)
    n = 20011
    box = 0.35 * np.array(mesh)
    r = np.mod(rng.uniform(0, 1, (n, 3)) * box, box)
    r[: n // 3] = np.mod(box / 2 + rng.normal(0, 0.4, (n // 3, 3)), box)
    r = torch.as_tensor(np.mod(r.astype(np.float32), box.astype(np.float32)), device="cuda")
    types = torch.as_tensor(rng.integers(0, T, n).astype(np.int32), device="cuda")
    charges = torch.as_tensor(rng.choice([-1.0, 0.0, 0.5], n).astype(np.float32), device="cuda")
    pm = ParticleMesh(mesh, box, T)
    A = rng.normal(size=(T, T))
    Q = A @ A.T + np.eye(T)
    _lib.call("hpf_ctx_set_functional", pm._h, _lib.dvec(Q.reshape(-1)), _lib.dvec([-1.0] * T),
              0.0, 0.4)
    masses = _lib.dvec(rng.uniform(0.5, 2.0, T))
    qt = _lib.dvec(rng.normal(size=T))
    got = {}
    for path in ("cufft", "fused", "fused"):
        pm.spectral = path
        out = torch.zeros(32, dtype=torch.float64, device="cuda")
        _lib.call("hpf_energy_fp64", pm._h, _lib.ptr(r), _lib.ptr(types), n, masses,
                  _lib.ptr(charges) if q else None, qt, 1.7, _lib.ptr(out), _lib.stream_ptr())
        got.setdefault(path, []).append(out.cpu().numpy())
    ref = got["cufft"][0]
    assert np.array_equal(got["fused"][0], got["fused"][1])
    for o in got["fused"]:
        assert np.allclose(o[:5], ref[:5], rtol=1e-11, atol=0)
        scale = np.abs(ref[5:9]).max() + np.sqrt(np.abs(ref[4] * ref[0])) + 1e-30
        assert np.abs(o[5:9] - ref[5:9]).max() <= 1e-11 * max(scale, np.abs(ref[6:9]).max())
        assert np.allclose(o[16:16 + T], ref[16:16 + T], rtol=1e-12, atol=0)
    pm.check_errors()

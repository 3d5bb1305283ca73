"""FP64 energy sums on the fused meshes hold 64-bit numbers throughout, as the
library-FFT path does.

- Beads on mesh points deposit exactly, so the densities are known as integers, and
  the sums can be compared with a direct transform in extended precision.  Two types
  fill one another's gaps (phi_A + phi_B uniform): under a Q whose large part is
  (phi_A + phi_B)^2 every mode's quadratic form cancels.  Each of a term's two factors
  carries about one rounding per level of its transform (log2 of the axis; the density
  varies along z alone) and some four more (filter, scales, Q, k^2), each at most
  2^-53, and the modes' errors are independent: (log2 nz + 4) 2^-53 of the sum of the
  terms' absolute values.
- In units where the sums lie outside FP32's exponents both paths agree to 1e-12."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _sums(pm, r, types, masses, path, q=None, qt=None, fac=0.0):
    from hymd_gb300 import _lib
    pm.spectral = path
    out = torch.zeros(32, dtype=torch.float64, device="cuda")
    _lib.call("hpf_energy_fp64", pm._h, _lib.ptr(r), _lib.ptr(types), r.shape[0],
              _lib.dvec(masses), _lib.ptr(q), _lib.dvec(qt) if qt is not None else None, fac,
              _lib.ptr(out), _lib.stream_ptr())
    pm.check_errors()
    return out.cpu().numpy()


@pytest.mark.parametrize("nz", [16, 48, 64, 128])
@pytest.mark.parametrize("inc", [2.5, 1.0e3])
@pytest.mark.parametrize("seed", range(4))
def test_exact_deposits(nz, inc, seed):
    from hymd_gb300 import _lib
    from hymd_gb300.field import ParticleMesh
    rng = np.random.default_rng(100 * nz + seed)
    n0 = 48 if nz == 48 else 16
    mesh = (n0, n0, nz)
    h, sigma, full = 0.5, 0.4, 5
    box = h * np.array(mesh)
    # per z plane: cA beads of A and full - cA of B on every mesh point
    cA = rng.integers(0, full + 1, nz)
    pts = np.stack(np.meshgrid(*[np.arange(k) for k in mesh], indexing="ij"), -1).reshape(-1, 3)
    r = np.repeat(pts, full, axis=0).astype(np.float32) * np.float32(h)
    types = (np.arange(full)[None, :] >= cA[pts[:, 2]][:, None]).astype(np.int32).reshape(-1)
    chi = 1.9
    Q = np.array([[inc, inc + chi], [inc + chi, inc]])
    pm = ParticleMesh(mesh, box, 2)
    _lib.call("hpf_ctx_set_functional", pm._h, _lib.dvec(Q.reshape(-1)), _lib.dvec([0.0, 0.0]),
              0.0, sigma)
    o = _sums(pm, torch.as_tensor(r, device="cuda"), torch.as_tensor(types, device="cuda"),
              [1.0, 1.0], "fused")
    # extended precision: modes (0, 0, kz), kz = 1 .. nz - 1
    ld = np.longdouble
    z, kz = np.arange(nz), np.arange(1, nz)
    arg = 2 * ld(np.pi) + ld("1.2246467991473531772e-16") * 2
    ph = arg / nz * ((z[:, None] * kz[None, :]) % nz).astype(ld)
    c, s = np.cos(ph), np.sin(ph)
    dV = ld(h) ** 3
    rho = [cA.astype(ld) / dV, (full - cA).astype(ld) / dV]
    re = [(x[:, None] * c).sum(0) / nz for x in rho]
    im = [(x[:, None] * s).sum(0) / nz for x in rho]
    k = arg / ld(box[2]) * np.where(kz > nz // 2, kz - nz, kz).astype(ld)
    H2 = np.exp(-(ld(sigma) * k) ** 2)
    pair = [[H2 * (re[i] * re[j] + im[i] * im[j]) for j in range(2)] for i in range(2)]
    term = sum(ld(Q[i, j]) * pair[i][j] for i in range(2) for j in range(2))
    size = sum(abs(ld(Q[i, j]) * pair[i][j]) for i in range(2) for j in range(2))
    tol = (np.log2(nz) + 4) * 2.0 ** -53
    for got, w in ((o[0], ld(1)), (o[3], k * k)):
        assert abs(ld(got) - (w * term).sum()) <= tol * (w * size).sum()


@pytest.mark.parametrize("unit", [1e-9, 1.0, 1e7])
def test_units_outside_fp32(unit):
    from hymd_gb300 import _lib
    from hymd_gb300.field import ParticleMesh
    rng = np.random.default_rng(5)
    n, mesh = 5000, (16, 16, 32)
    box = 0.4 * unit * np.array(mesh)
    r = torch.as_tensor((rng.uniform(0, 0.999, (n, 3)) * box).astype(np.float32), device="cuda")
    types = torch.as_tensor(rng.integers(0, 2, n).astype(np.int32), device="cuda")
    q = torch.as_tensor(rng.choice([-1.0, 0.0, 1.0], n).astype(np.float32), device="cuda")
    pm = ParticleMesh(mesh, box, 2)
    Q = np.array([[2.0, 1.5], [1.5, 2.0]])
    _lib.call("hpf_ctx_set_functional", pm._h, _lib.dvec(Q.reshape(-1)), _lib.dvec([0.0, 0.0]),
              0.0, 0.5 * unit)
    args = (pm, r, types, [0.7, 1.3])
    a = _sums(*args, "fused", q, [0.3, -0.2], 1.7)
    b = _sums(*args, "cufft", q, [0.3, -0.2], 1.7)
    assert np.all(np.isfinite(a[:9])) and np.all(b[:5] != 0)
    assert np.allclose(a[:5], b[:5], rtol=1e-12, atol=0)
    assert np.allclose(a[5], b[5], rtol=1e-12, atol=0)
    # (the weighted cross sums cancel further)
    assert np.allclose(a[6:9], b[6:9], rtol=1e-10, atol=1e-12 * np.abs(b[6:9]).max())
    assert np.allclose(a[16:18], b[16:18], rtol=1e-13, atol=0)

"""The one-launch density profile (hpf_z_profile) and its gradient against the
tensor-operation form in 64 bits: one bead, one bin, bins in shared and in
global memory, beads on bin edges and on the box faces.

Weights are rounded to 2^-24 of a bead and the coordinates are FP32 (1e-7 of
the box, times n_bins in the bin fraction): profile within (1 + n_bins) 2e-7
per bead of a bin, gradients within 1e-6 of their size except where FP32 and
FP64 disagree on which side of a bin centre a bead lies (both are derivatives
there).  Also the functional set from chi on the device against the one set
from the host."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,T,bins", [(1, 1, 1), (255, 2, 7), (5000, 5, 100), (20001, 3, 4001)])
def test_profile_and_gradient(n, T, bins):
    from hymd_gb300.reverse import _z_profile_torch, z_profile
    rng = np.random.default_rng(n)
    box = [3.0, 4.0, 5.5]
    z = rng.uniform(0, box[2], n)
    z[: n // 10] = np.round(z[: n // 10] / box[2] * bins) * box[2] / bins  # bin edges
    x = np.stack([rng.uniform(0, 3, n), rng.uniform(0, 4, n), z], 1).astype(np.float32)
    types = torch.as_tensor(rng.integers(0, T, n).astype(np.int32), device="cuda")
    g = torch.as_tensor(rng.normal(size=(T, bins)).astype(np.float32), device="cuda")
    a = torch.as_tensor(x, device="cuda").requires_grad_(True)
    b = torch.as_tensor(x, device="cuda").double().requires_grad_(True)
    pa, pb = z_profile(a, types, T, bins, box), _z_profile_torch(b, types, T, bins, box)
    vol = box[0] * box[1] * box[2] / bins
    tol = 2e-7 * (1 + bins) * (pb * vol + 1) / vol
    assert bool(((pa.double() - pb).abs() <= tol).all())
    assert torch.equal(pa, z_profile(a, types, T, bins, box))
    (ga,) = torch.autograd.grad(pa, a, g, create_graph=False)
    (gb,) = torch.autograd.grad(pb, b, g.double())
    s = b.detach()[:, 2] * (bins / box[2]) - 0.5
    clear = (s - s.round()).abs() > 1e-6 * bins
    scale = float(gb.abs().max()) + 1e-30
    assert float((ga.double() - gb)[clear].abs().max() if clear.any() else 0.0) <= 1e-6 * scale
    assert float(ga[:, :2].abs().max()) == 0.0
    # derivatives of derivatives: linear in the incoming gradient
    gr = g.clone().requires_grad_(True)
    (g1,) = torch.autograd.grad(z_profile(a, types, T, bins, box), a, gr, create_graph=True)
    (g2,) = torch.autograd.grad(g1.sum(), gr)
    assert g2.shape == gr.shape


def test_profile_non_finite():
    from hymd_gb300.reverse import z_profile
    x = torch.rand(100, 3, device="cuda")
    x[17, 2] = float("nan")
    t = torch.zeros(100, dtype=torch.int32, device="cuda")
    assert bool(torch.isnan(z_profile(x, t, 1, 10, [1.0, 1.0, 1.0])).any())


@pytest.mark.parametrize("kind", ["DefaultWithChi", "DefaultNoChi", "SquaredPhi"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_functional_from_chi(kind, dtype):
    from hymd_gb300 import _lib
    from hymd_gb300.adjoint import functional_coefficients
    from hymd_gb300.field import ParticleMesh
    T, n = 3, 4000
    chi = torch.randn(T, T, dtype=dtype, device="cuda") * 10
    pm = ParticleMesh([24] * 3, [6.0] * 3, T)
    r = torch.rand(n, 3, device="cuda") * 6
    types = (torch.arange(n, device="cuda") % T).int()
    out = []
    for dev in (False, True):
        if dev:
            _lib.call("hpf_ctx_set_functional_chi", pm._h, _lib.ptr(chi),
                      int(dtype == torch.float64), int(kind == "DefaultWithChi"), 0.05, 8.3,
                      0.0 if kind == "SquaredPhi" else 8.1, 0.5, _lib.stream_ptr())
        else:
            Q, b, c = functional_coefficients(kind, chi.cpu().numpy(), 0.05, 8.3, 8.1)
            _lib.call("hpf_ctx_set_functional", pm._h, _lib.dvec(Q.reshape(-1)), _lib.dvec(b),
                      float(c), 0.5)
        F = torch.zeros_like(r)
        _lib.call("hpf_field_step", pm._h, _lib.ptr(r), _lib.ptr(types), n, _lib.dvec([1.0] * T),
                  _lib.ptr(F), None, None, None, _lib.stream_ptr())
        out.append(F.clone())
    assert float((out[0] - out[1]).abs().max()) <= 1e-6 * float(out[0].abs().max())

"""The charge force's vector-Jacobian product on contexts of one to eight types (which
differ in the transform batches they have plans for) against torch's FP64 autograd, on a
library-FFT mesh and on a fused one."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import torch_field as tf  # noqa: E402


@pytest.mark.parametrize("mesh", [(18, 20, 22), (16, 16, 16)])
@pytest.mark.parametrize("T", [1, 2, 3, 5, 8])
def test_types(mesh, T):
    from hymd_gb300 import _lib
    from hymd_gb300.field import ParticleMesh
    rng = np.random.default_rng(T)
    n, box, sigma = 2000, 0.4 * np.array(mesh), 0.5
    r = torch.as_tensor((rng.uniform(0, 0.999, (n, 3)) * box).astype(np.float32), device="cuda")
    q = torch.as_tensor(rng.choice([-1.0, 0.0, 1.0], n).astype(np.float32), device="cuda")
    lam = torch.as_tensor(rng.normal(size=(n, 3)).astype(np.float32), device="cuda")
    pm = ParticleMesh(mesh, box, T)
    _lib.call("hpf_ctx_set_functional", pm._h, _lib.dvec(np.eye(T).reshape(-1)),
              _lib.dvec([0.0] * T), 0.0, sigma)
    g = torch.empty_like(r)
    _lib.call("hpf_pic_force_vjp", pm._h, _lib.ptr(r), _lib.ptr(q), n, 1.7, _lib.ptr(lam),
              _lib.ptr(g), _lib.stream_ptr())
    y = r.double().clone().requires_grad_(True)
    E = tf.pic_force(y, q.double(), list(mesh), list(box), sigma, 1.7)
    (lam.double() * E).sum().backward()
    err = (g.double() - y.grad).norm() / y.grad.norm()
    assert float(err) < 1e-4
    pm.check_errors()

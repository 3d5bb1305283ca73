"""FP64 energies recorded in a graph after a first evaluation outside it: a charged
one after an uncharged one and the other way round, on a library-FFT mesh and on a
fused one, and after a change of the spectral path.  The replay has the bits of the
same call made eagerly."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

T, N = 2, 3000


def _energy(pm, r, types, q, out):
    from hymd_gb300 import _lib
    _lib.call("hpf_energy_fp64", pm._h, _lib.ptr(r), _lib.ptr(types), N, _lib.dvec([1.0] * T),
              _lib.ptr(q), _lib.dvec([0.3, -0.2]), 1.7, _lib.ptr(out), _lib.stream_ptr())


@pytest.mark.parametrize("mesh,paths", [
    ((10, 12, 14), ("cufft", "cufft")), ((16, 16, 16), ("fused", "fused")),
    ((16, 16, 16), ("fused", "cufft")), ((16, 16, 16), ("cufft", "fused"))])
@pytest.mark.parametrize("first_charged", [False, True])
def test_capture_after_the_other(mesh, paths, first_charged):
    from hymd_gb300 import _lib
    from hymd_gb300.field import ParticleMesh
    rng = np.random.default_rng(8)
    r = torch.as_tensor((rng.uniform(0, 0.999, (N, 3)) * 6).astype(np.float32), device="cuda")
    types = (torch.arange(N, device="cuda") % T).int()
    q = torch.as_tensor(rng.choice([-1.0, 0.0, 1.0], N).astype(np.float32), device="cuda")

    def make():
        pm = ParticleMesh(mesh, [6.0] * 3, T)
        _lib.call("hpf_ctx_set_functional", pm._h, _lib.dvec([2.0, 1.5, 1.5, 2.0]),
                  _lib.dvec([-1.0] * T), 0.5, 0.4)
        return pm

    first, second = (q, None) if first_charged else (None, q)
    out = torch.zeros(32, dtype=torch.float64, device="cuda")
    ref = make()
    if paths[1] != ref.spectral:
        ref.spectral = paths[1]
    _energy(ref, r, types, second, out)
    want = out.clone()
    pm = make()
    if paths[0] != pm.spectral:
        pm.spectral = paths[0]
    _energy(pm, r, types, first, out)
    if paths[1] != pm.spectral:
        pm.spectral = paths[1]
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        _energy(pm, r, types, second, out)
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out[:16 + T], want[:16 + T])
    pm.check_errors()

"""ForceModel.set_chi on the host path sends the functional again whenever another
call on the same mesh has set one since (update_field, field_energy, another
ForceModel), and not when its own is still in place.  No GPU: the calls are counted."""
import types

import pytest

torch = pytest.importorskip("torch")


def _model(pm):
    from hymd_gb300.reverse import ForceModel
    m = ForceModel.__new__(ForceModel)
    m.pm, m.T, m.kind = pm, 2, "DefaultWithChi"
    m.kappa, m.rho0, m.a, m.sigma = 0.05, 8.0, 8.0, 0.5
    return m


def test_host_functional_is_sent_again(monkeypatch):
    from hymd_gb300 import _lib, adjoint
    sent = []
    monkeypatch.setattr(_lib, "call", lambda name, *a: sent.append(name))
    monkeypatch.setattr(_lib, "stream_ptr", lambda *a: None)
    pm = types.SimpleNamespace(_h=None, _functional=None)
    a, b = _model(pm), _model(pm)
    chi, other = torch.eye(2) + 3.0, torch.eye(2) - 7.0
    a.set_chi(chi)
    a.set_chi(chi)
    assert len(sent) == 1
    b.set_chi(other)
    a.set_chi(chi)
    assert len(sent) == 3
    Q, bb, c = adjoint.functional_coefficients("DefaultWithChi", other.numpy(), 0.05, 8.0, 8.0)
    adjoint._set(pm, Q, bb, c, 0.5)
    a.set_chi(chi)
    assert len(sent) == 5
    pm._functional = ("another", "functional")  # as ParticleMesh.set_functional leaves it
    a.set_chi(chi)
    a.set_chi(chi)
    assert len(sent) == 6

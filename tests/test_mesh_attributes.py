"""What a mesh context offers and keeps alive, without a GPU: the scratch spectra of
before under their names, allocated when asked for, and one table of meshes."""
import gc
import weakref

import pytest

torch = pytest.importorskip("torch")


def _pm():
    from hymd_gb300.field import ParticleMesh
    pm = ParticleMesh.__new__(ParticleMesh)
    pm._h, pm.Nmesh, pm.n_types, pm.device = None, (4, 6, 8), 2, torch.device("cpu")
    return pm


def test_scratch_spectra():
    pm = _pm()
    assert pm.spec_raw.shape == (2, 4, 6, 5) and pm.spec_raw.dtype == torch.complex64
    assert pm.spec_force.shape == (6, 4, 6, 5) and pm.spec_force.dtype == torch.complex64
    assert pm.spec_raw is pm.spec_raw and pm.spec_force is pm.spec_force


def test_one_table_of_meshes():
    from hymd_gb300 import field
    pm = _pm()
    k = torch.zeros(1, dtype=torch.complex64)
    pm.fields = dict(phi_fourier=k)
    field._REGISTRY[-1] = pm
    field._REGISTRY_FOURIER[k.data_ptr()] = pm
    assert field._pm_of_fourier([k]) is pm
    # a mesh taken out of the table is given back
    gone = weakref.ref(pm)
    del field._REGISTRY[-1], pm
    gc.collect()
    assert gone() is None
    with pytest.raises(ValueError):
        field._pm_of_fourier([k])

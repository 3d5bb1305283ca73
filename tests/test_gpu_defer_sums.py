"""The rRESPA sums run beside the field step's first pass (hpf_respa_plan_defer)
or in stream order: the same kernels on the same inputs, so every result is
bit-identical, eager and captured.  With a barostat, whose box update the pass
needs, they stay in stream order."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,mesh,npt", [("melt", 16, False), ("melt", 24, False),
                                           ("membrane", 24, False), ("membrane", 32, True)])
def test_deferred_sums_are_identical(kind, mesh, npt):
    from hymd_gb300 import systems
    from hymd_gb300.hamiltonian import get_hamiltonian
    from hymd_gb300.md import RespaMD

    class InLine(RespaMD):
        _defer_sums = False

    if kind == "melt":
        s = systems.homopolymer_melt(seed=4, n_chains=150, length=10, box=5.6, mesh=mesh)
    else:
        s = systems.lipid_membrane(seed=9, n_lipids=60, n_water=900, box=5.6, mesh=mesh)
    out = []
    for cls in (RespaMD, InLine):
        md = cls(s["positions"], s["velocities"], s["types"], s["config"],
                 get_hamiltonian(s["config"]), topology=s["topology"], max_block_beads=24)
        md.TUNE_SPECTRAL_TILE = False
        md.couple(thermostat=True, barostat="isotropic" if npt else None, seed=3,
                  n_steps=30)
        md.prime()
        md.run(3)
        md.capture()
        md.run(5)
        torch.cuda.synchronize()
        md.check_errors()
        out.append(md)
    assert out[0]._defer_sums == (not npt) and not out[1]._defer_sums
    for name in ("r", "v", "f_b", "f_field", "box", "bonded_out", "state", "field_sums"):
        assert torch.equal(getattr(out[0], name), getattr(out[1], name)), name

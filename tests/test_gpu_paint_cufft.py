"""Deposits made by the rRESPA launch on meshes of the library-FFT path (ragged,
odd, a single odd axis) against the separate paint: the same integers, so
every result is bit-identical, eager and captured; charged systems keep the
separate paint."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,mesh", [("melt", [20, 18, 21]), ("melt", [16, 16, 18]),
                                       ("charged", [20, 21, 22]), ("charged", [25, 25, 25])])
def test_fused_paint_is_identical(kind, mesh):
    from hymd_gb300 import systems
    from hymd_gb300.hamiltonian import get_hamiltonian
    from hymd_gb300.md import RespaMD

    class Separate(RespaMD):
        FUSE_PAINT = False

    if kind == "melt":
        s = systems.homopolymer_melt(seed=4, n_chains=150, length=10, box=5.6, mesh=mesh)
    else:
        s = systems.charged_peptides(seed=8, n_chains=6, n_res=20, n_total=4000, box=7.5, mesh=mesh)
    out = []
    for cls in (RespaMD, Separate):
        md = cls(s["positions"], s["velocities"], s["types"], s["config"],
                 get_hamiltonian(s["config"]), topology=s["topology"], charges=s.get("charges"),
                 max_block_beads=32)
        md.couple(thermostat=True, seed=3, n_steps=30)
        md.prime()
        md.run(2)
        md.capture()
        md.run(3)
        torch.cuda.synchronize()
        md.check_errors()
        out.append(md)
    assert out[0].pm.spectral == "cufft"
    assert out[0]._paint_fused == (kind == "melt") and not out[1]._paint_fused
    names = ["r", "v", "f_b", "f_field", "bonded_out"] + (["f_elec"] if kind == "charged" else [])
    for name in names:
        assert torch.equal(getattr(out[0], name), getattr(out[1], name)), name

"""The drop-in update_field and update_field_force_q on the fused spectral
passes against the cuFFT path: filtered densities, spectra, force mesh,
external potentials and charge grids, at the smallest and largest lengths, 3 *
2^a, one to five types (more fall back to cuFFT where the tile does not fit),
twice in a row.  Both are FP32 transforms of the same deposits: 1e-6 relative
RMS per grid (their errors against 64 bits are 1e-7 to 5e-7)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _rel(a, b):
    a, b = (torch.view_as_real(t) if t.is_complex() else t for t in (a, b))
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize("mesh,T", [
    ((8, 16, 16), 1), ((16, 16, 32), 2), ((32, 64, 16), 3), ((24, 24, 24), 4),
    ((96, 48, 48), 2), ((256, 16, 16), 2), ((64, 64, 64), 8), ((16, 128, 128), 5),
    ((192, 24, 24), 5)])
def test_matches_cufft(mesh, T):
    from hymd_gb300 import field as gf
    from hymd_gb300.config import Config
    from hymd_gb300.force import Chi
    from hymd_gb300.hamiltonian import get_hamiltonian
    rng = np.random.default_rng(sum(mesh) + T)
    n = 9001
    box = 0.4 * np.array(mesh)
    r = torch.as_tensor((rng.uniform(0, 0.999, (n, 3)) * box).astype(np.float32), device="cuda")
    types = torch.as_tensor(rng.integers(0, T, n).astype(np.int32), device="cuda")
    q = torch.as_tensor(rng.choice([-1.0, 0.0, 1.0], n).astype(np.float32), device="cuda")
    names = [chr(65 + i) for i in range(T)]
    cfg = Config(n_steps=1, time_step=0.03, mesh_size=list(mesh), sigma=0.5, kappa=0.05,
                 box_size=box, n_particles=n, n_types=T, mass=72.0, hamiltonian="DefaultWithChi",
                 unique_names=names, type_to_name_map=dict(enumerate(names)),
                 chi=[Chi(names[i], names[i + 1], 9.0) for i in range(T - 1)],
                 m=[1.0 + 0.25 * t for t in range(T)], coulombtype="PIC_Spectral",
                 dielectric_const=15.0)
    ham = get_hamiltonian(cfg)
    pm, fields, elec, coulomb = gf.initialize_pm(None, cfg)
    phi, phi_k, fmesh, vk, v_ext, ptr, plap = fields
    phi_q, phi_qk, psi, ef = elec
    ef_k, psi_k = coulomb
    F, Fq = torch.zeros_like(r), torch.zeros_like(r)
    out = []
    for path in ("cufft", "fused", "fused"):
        pm.spectral = path
        for t in [*phi, *phi_k, *v_ext, phi_q, psi, psi_k, *ef, *(x for m in fmesh for x in m)]:
            t.fill_(7.0)
        gf.update_field(phi, plap, ptr, None, fmesh, ham, pm, r, types, cfg, v_ext, phi_k, vk,
                        cfg.m, compute_potential=True)
        gf.compute_field_force(None, r, fmesh, F, types, T)
        gf.update_field_force_q(q, phi_q, phi_qk, psi, psi_k, ef_k, ef, Fq, None, ham, pm, r, cfg)
        torch.cuda.synchronize()
        pm.check_errors()
        out.append([t.clone() for t in (*phi, *phi_k, *v_ext, phi_q, psi, psi_k, *ef,
                                        *(x for m in fmesh for x in m), F, Fq)])
    for ref, a, b in zip(*out):
        assert torch.equal(a, b)
        assert _rel(a, ref) < 1e-6

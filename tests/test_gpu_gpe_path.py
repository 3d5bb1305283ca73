"""The variable-dielectric solve after a change of the spectral path on one context:
the loop graph follows the path (the same results as a context that never had another
one), and a repeated solve, which replays the cached graph, has the same bits."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_loop_follows_the_path():
    from hymd_gb300 import field as gf
    from hymd_gb300.config import Config
    from hymd_gb300.hamiltonian import get_hamiltonian
    rng = np.random.default_rng(3)
    T, mesh = 3, (24, 24, 24)
    box = 0.3 * np.array(mesh)
    n = int(8 * np.prod(box))
    r = torch.as_tensor((rng.uniform(0, 0.999, (n, 3)) * box).astype(np.float32), device="cuda")
    types = torch.as_tensor(rng.integers(0, T, n).astype(np.int32), device="cuda")
    q = torch.as_tensor(rng.choice([-1.0, 0.0, 0.0, 1.0], n).astype(np.float32), device="cuda")
    cfg = Config(n_steps=1, time_step=0.03, mesh_size=list(mesh), sigma=0.5, kappa=0.05,
                 box_size=box, n_particles=n, n_types=T, mass=72.0, hamiltonian="DefaultNoChi",
                 m=[1.0] * T, coulombtype="PIC_Spectral_GPE", type_charges=[0.3, -0.2, 0.0],
                 dielectric_type=[80.0, 5.0, 20.0], conv_crit=1e-5, pol_mixing=0.6,
                 convergence_type="max_diff")
    ham = get_hamiltonian(cfg)

    def solves(paths):
        pm, fields, elec, coulomb = gf.initialize_pm(None, cfg)
        phi, phi_k, fmesh, vk, v_ext, ptr, plap = fields
        phi_q, phi_qk, psi, ef = elec
        eps, epsk, eta, etak, pol, pol_prev, _, contrib, vbar, vbark, fme, fmek = coulomb
        out = []
        for path in paths:
            # the densities come from the fused path each time
            pm.spectral = "fused"
            gf.update_field(phi, plap, ptr, None, fmesh, ham, pm, r, types, cfg, v_ext, phi_k, vk,
                            cfg.m)
            pm.spectral = path
            pol_prev.zero_()
            F = torch.zeros_like(r)
            vb, e, dot = gf.update_field_force_q_GPE(
                None, phi, types, q, phi_q, phi_qk, eps, epsk, eta, etak, pol_prev, pol, ef, F,
                contrib, psi, vbar, vbark, fme, fmek, ham, None, None, pm, r, cfg)
            torch.cuda.synchronize()
            pm.check_errors()
            out.append([x.clone() for x in (*vb, e, dot, psi, *ef, F, pol)])
        return out

    (cufft,), (fused,) = solves(["cufft"]), solves(["fused"])
    assert not all(torch.equal(a, b) for a, b in zip(cufft, fused))
    got = solves(["cufft", "fused", "fused", "cufft", "cufft"])
    for out, want in zip(got, (cufft, fused, fused, cufft, cufft)):
        for a, b in zip(out, want):
            assert torch.equal(a, b)

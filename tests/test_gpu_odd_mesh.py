"""Meshes with an odd number of points: grids of one stack then start on odd multiples of
four bytes, where the transform library wants eight.  The variable-dielectric solve, the
force's vector-Jacobian product, the charge chain and single transforms of a stack's
grids against the FP64 oracle and its torch form, with the bounds of the same tests on
even meshes."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import field as of  # noqa: E402
from oracle import hamiltonian as oh  # noqa: E402
from oracle import torch_field as tf  # noqa: E402


def rel_rms(a, b):
    a = np.asarray(a, np.float64)
    b = np.asarray(b, np.float64)
    return float(np.sqrt(np.mean((a - b) ** 2)) / np.sqrt(np.mean(b ** 2)))


def _config(mesh, rng):
    from hymd_gb300.config import Config
    from hymd_gb300.force import Chi
    T, n = 3, 3000
    box = np.array([5.0, 5.0, 5.5])
    r = rng.uniform(0, 1, (n, 3)) * box
    r[: n // 3] = np.mod(box / 2 + rng.normal(0, 0.6, (n // 3, 3)), box)
    r = np.mod(r.astype(np.float32), box.astype(np.float32))
    types = rng.integers(0, T, n).astype(np.int32)
    q = np.zeros(n, np.float32)
    k = rng.permutation(n)[: n // 5]
    q[k] = rng.choice([-1.0, 1.0], len(k)).astype(np.float32)
    names = ["A", "B", "C"]
    chi = [Chi("A", "B", 12.0), Chi("A", "C", 4.0), Chi("B", "C", 20.0)]
    cfg = Config(n_steps=1, time_step=0.03, mesh_size=list(mesh), sigma=0.5, kappa=0.05,
                 box_size=box, n_particles=n, n_types=T, mass=72.0,
                 hamiltonian="DefaultWithChi", unique_names=names,
                 type_to_name_map=dict(enumerate(names)), chi=chi, m=[1.0, 1.0, 1.0],
                 coulombtype="PIC_Spectral_GPE", type_charges=[0.3, -0.3, 0.0],
                 dielectric_type=[80.0, 2.0, 10.0], conv_crit=1e-7, pol_mixing=0.6,
                 convergence_type="max_diff")
    return cfg, r, types, q


@pytest.mark.parametrize("mesh", [(23, 25, 27), (19, 19, 19)])
def test_gpe(mesh):
    from hymd_gb300 import field as gf
    from hymd_gb300.hamiltonian import get_hamiltonian
    cfg, r, types, q = _config(mesh, np.random.default_rng(21))
    T = cfg.n_types
    ham = get_hamiltonian(cfg)
    pm, fl, ecl, cl = gf.initialize_pm(None, cfg)
    phi, phi_k, fmesh, vk, v_ext, ptr, plap = fl
    phi_q, phi_qk, psi, ef = ecl
    eps, epsk, eta, etak, pol, pol_prev, _, contrib, vbar, vbark, fme, fmek = cl
    R, Ty, Qc = (torch.as_tensor(a, device="cuda") for a in (r, types, q))
    gf.update_field(phi, plap, ptr, None, fmesh, ham, pm, R, Ty, cfg, v_ext, phi_k, vk, cfg.m)
    chim = np.zeros((T, T))
    for c in cfg.chi:
        i, j = cfg.unique_names.index(c.atom_1), cfg.unique_names.index(c.atom_2)
        chim[i, j] = chim[j, i] = c.interaction_energy
    fun = oh.quadratic_from_params("DefaultWithChi", T, cfg.kappa, cfg.rho0, cfg.a, chim)
    ref_field = of.update_field(r.astype(np.float64), types, T, cfg.mesh(), cfg.box(), cfg.m,
                                fun, cfg.sigma)
    zero = lambda: np.zeros(tuple(cfg.mesh()))  # noqa: E731
    ref = of.gpe_step(ref_field["phi"], q, r, types, T, cfg.mesh(), cfg.box(), cfg.sigma,
                      cfg.dielectric_type, cfg.type_charges,
                      dict(phi_eps=zero(), pol_prev=zero(), contrib=zero()),
                      conv_crit=cfg.conv_crit, mixing=cfg.pol_mixing, conv_kind="max_diff")
    F = torch.zeros_like(R)
    for _ in range(2):
        vb, e, dot = gf.update_field_force_q_GPE(
            None, phi, Ty, Qc, phi_q, phi_qk, eps, epsk, eta, etak, pol_prev, pol, ef, F, contrib,
            psi, vbar, vbark, fme, fmek, ham, None, None, pm, R, cfg)
        assert abs(pm.gpe_iterations - ref["iterations"]) <= 2
        assert rel_rms(e.cpu().numpy(), ref["phi_eps"]) < 1e-6
        assert rel_rms(psi.cpu().numpy(), ref["psi"]) < 1e-4
        assert rel_rms(torch.stack(list(ef)).cpu().numpy(), ref["elec_field"]) < 1e-4
        assert rel_rms(F.cpu().numpy(), ref["forces"]) < 1e-4
        assert rel_rms(torch.stack(list(vb)).cpu().numpy(), ref["Vbar"]) < 1e-4
    pm.check_errors()


@pytest.mark.parametrize("mesh,T", [((19, 21, 23), 2), ((19, 21, 23), 3), ((17, 17, 17), 1),
                                    ((17, 17, 17), 5)])
def test_force_vjps(mesh, T):
    from hymd_gb300 import _lib
    from hymd_gb300.field import ParticleMesh
    rng = np.random.default_rng(T)
    n, box, sigma = 2000, 0.4 * np.array(mesh), 0.5
    r = torch.as_tensor((rng.uniform(0, 0.999, (n, 3)) * box).astype(np.float32), device="cuda")
    types = torch.as_tensor(rng.integers(0, T, n).astype(np.int32), device="cuda")
    q = torch.as_tensor(rng.choice([-1.0, 0.0, 1.0], n).astype(np.float32), device="cuda")
    lam = torch.as_tensor(rng.normal(size=(n, 3)).astype(np.float32), device="cuda")
    A = rng.normal(size=(T, T))
    Q = A @ A.T + np.eye(T)
    pm = ParticleMesh(mesh, box, T)
    _lib.call("hpf_ctx_set_functional", pm._h, _lib.dvec(Q.reshape(-1)), _lib.dvec([0.0] * T),
              0.0, sigma)
    g, gp = torch.empty_like(r), torch.empty_like(r)
    dQ = torch.zeros(T * T, dtype=torch.float64, device="cuda")
    _lib.call("hpf_field_force_vjp", pm._h, _lib.ptr(r), _lib.ptr(types), n, _lib.dvec([1.0] * T),
              _lib.ptr(lam), _lib.ptr(g), _lib.ptr(dQ), _lib.stream_ptr())
    _lib.call("hpf_pic_force_vjp", pm._h, _lib.ptr(r), _lib.ptr(q), n, 1.7, _lib.ptr(lam),
              _lib.ptr(gp), _lib.stream_ptr())
    x = r.double().clone().requires_grad_(True)
    Qt = torch.as_tensor(Q, device="cuda").requires_grad_(True)
    F = tf.field_force(x, types, T, [1.0] * T, list(mesh), list(box), Qt, sigma)
    (lam.double() * F).sum().backward()
    assert rel_rms(g.cpu().numpy(), x.grad.cpu().numpy()) < 1e-4
    assert rel_rms(dQ.cpu().numpy(), Qt.grad.reshape(-1).cpu().numpy()) < 1e-4
    y = r.double().clone().requires_grad_(True)
    E = tf.pic_force(y, q.double(), list(mesh), list(box), sigma, 1.7)
    (lam.double() * E).sum().backward()
    assert rel_rms(gp.cpu().numpy(), y.grad.cpu().numpy()) < 1e-4
    pm.check_errors()


@pytest.mark.parametrize("first", [0, 1, 2])
def test_transforms_of_a_part_of_a_stack(first):
    """hpf_r2c / hpf_c2r on grids first .. of a stack, against torch's FP64 transforms."""
    from hymd_gb300 import _lib
    from hymd_gb300.field import ParticleMesh
    mesh, T = (9, 11, 13), 2
    pm = ParticleMesh(mesh, [4.0] * 3, T)
    gen = torch.Generator(device="cuda").manual_seed(first)
    x = torch.randn(5, *mesh, generator=gen, device="cuda")
    spec = pm.complex_field(T)
    part = x[first:first + T]
    _lib.call("hpf_r2c", pm._h, _lib.ptr(part), _lib.ptr(spec), T, _lib.stream_ptr())
    want = torch.fft.rfftn(part.double(), dim=(1, 2, 3))
    assert float((spec - want).abs().max()) <= 1e-5 * float(want.abs().max())
    y = torch.full((5, *mesh), 7.0, device="cuda")
    keep = spec.clone()
    _lib.call("hpf_c2r", pm._h, _lib.ptr(spec), _lib.ptr(y[first:]), T, _lib.stream_ptr())
    back = torch.fft.irfftn(keep.to(torch.complex128), s=mesh, dim=(1, 2, 3)) * np.prod(mesh)
    assert float((y[first:first + T] - back).abs().max()) <= 1e-5 * float(back.abs().max())
    rest = torch.cat([y[:first], y[first + T:]])
    assert bool((rest == 7.0).all())

"""Reverse mode of the fused inner loop (hpf_respa_vjp) against the
step-by-step form (per-step kicks, drifts and bonded forces as separate
differentiable operations): lane-sized groups, warp groups, chains of one CTA,
with and without four-body terms, with free beads, and a plan of nothing but
one molecule.

Both are FP32 with the same Jacobian-vector products summed in another order:
over 3 inner steps the gradients agree to a few times the 1e-6 of a single
product, amplified by the stiff bonds (dt^2 k / m ~ 0.02 a step): 2e-5
relative RMS."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(torch.sqrt((a - b).double().square().mean())
                 / torch.sqrt(b.double().square().mean()))


@pytest.mark.parametrize("kind,cap", [("melt", 10), ("melt", 32), ("melt", 64),
                                      ("membrane", 24), ("membrane", 64), ("one", 64),
                                      ("peptide16", 64), ("peptide80", 64), ("peptide16", 128)])
def test_matches_step_by_step(kind, cap):
    from hymd_gb300 import systems
    from hymd_gb300.hamiltonian import get_hamiltonian
    from hymd_gb300.md import RespaMD
    from hymd_gb300.reverse import ForceModel, _InnerLoop, bonded_force
    if kind == "melt":
        s = systems.homopolymer_melt(seed=4, n_chains=33, length=10, box=5.6, mesh=16)
    elif kind == "one":
        s = systems.homopolymer_melt(seed=4, n_chains=1, length=7, box=5.6, mesh=16)
    elif kind == "membrane":
        s = systems.lipid_membrane(seed=9, n_lipids=41, n_water=301, box=5.6, mesh=16)
    else:
        s = systems.charged_peptides(seed=5, n_chains=5, n_res=int(kind[7:]) // 2, n_total=1000,
                                     box=8.0, mesh=16)
        rng = np.random.default_rng(2)
        s["positions"] = np.mod(s["positions"] + rng.normal(0, 0.02, s["positions"].shape),
                                8.0).astype(np.float32)
    cfg = s["config"]
    cfg.barostat, cfg.respa_inner, cfg.time_step = None, 3, 0.01
    md = RespaMD(s["positions"], s["velocities"], s["types"], cfg, get_hamiltonian(cfg),
                 topology=s["topology"], max_block_beads=cap)
    model = ForceModel(md)
    assert model.fused_inner
    g = torch.Generator(device="cuda").manual_seed(1)
    rnd = lambda: torch.randn(md.n, 3, generator=g, device="cuda")  # noqa: E731
    leaves = [md.r.clone(), md.v.clone(), 20.0 * rnd(), bonded_force(md.r.clone(), model).detach()]
    cot = [rnd(), rnd(), 0.01 * rnd()]
    bonded = (leaves[3].abs().sum(1) > 0).float()[:, None]
    cot[2] = cot[2] * bonded  # (a free bead's force is zero and goes nowhere)
    m, dt, n_in = md.mass, md.dt, md.respa

    def steps(x, v, fs, fb):
        v = v + (0.5 * n_in * dt / m) * fs
        for _ in range(n_in):
            v = v + (0.5 * dt / m) * fb
            x = torch.remainder(x + dt * v, model.box_f)
            fb = bonded_force(x, model)
            v = v + (0.5 * dt / m) * fb
        return x, v, fb

    out = []
    for fn in (lambda *a: _InnerLoop.apply(*a, model), steps):
        ins = [t.clone().requires_grad_(True) for t in leaves]
        res = fn(*ins)
        grads = torch.autograd.grad(res, ins, cot)
        out.append((res, grads))
    (ra, ga), (rb, gb) = out
    assert _rel(ra[1], rb[1]) < 1e-5
    for k in range(3):
        assert _rel(ga[k], gb[k]) < 2e-5, k
    assert _rel(ga[3] * bonded, gb[3] * bonded) < 2e-5
    # no need for it: gradients of a subset, cotangents left out
    ins = [t.clone().requires_grad_(i == 2) for i, t in enumerate(leaves)]
    x, v, fb = _InnerLoop.apply(*ins, model)
    (gs,) = torch.autograd.grad((x * cot[0]).sum(), [ins[2]])
    ins2 = [t.clone().requires_grad_(i == 2) for i, t in enumerate(leaves)]
    (gs2,) = torch.autograd.grad((steps(*ins2)[0] * cot[0]).sum(), [ins2[2]])
    assert _rel(gs, gs2) < 2e-5
    md.check_errors()

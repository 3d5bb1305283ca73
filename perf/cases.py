"""The work that users of hymd_gb300 have it do, as cases for timing.

Kinds of case (`kind`) and the public entry points they go through:

  md        one outer rRESPA step of a running simulation (`RespaMD.run(1)`
            on the captured step): thermostat, and barostat or PIC_Spectral
            electrostatics where the system has them
  replicas  one outer step of a batch of small independent systems
            (`ReplicaBatch.run(1)`)
  field     the slow forces of one step through the drop-in calls of a
            HyMD-style main loop: `update_field`, `compute_field_force` and,
            with charges, `update_field_force_q`
  gpe       a variable-dielectric solve, `update_field_force_q_GPE`
  bonded    the bonded forces of one inner step through the drop-in calls
            `compute_bond_forces`, `compute_angle_forces`,
            `compute_dihedral_forces`
  report    energies and pressure at a print step:
            `compute_field_and_kinetic_energy` and `comp_pressure`
  adjoint   field energy and its gradients in the positions and chi
            (`field_energy`, forward and backward)
  reverse   a short differentiated trajectory (`profile_loss`, forward and
            backward: gradients in positions, velocities and chi)

Systems are the recipes of hymd_gb300.systems (melt of homopolymers, lipid
membrane in water, charged peptides in water) at the sizes of the
repository's own benchmarks and tests and between them; meshes have the
spacing of 0.3 to 0.5 nm that the field method wants, on power-of-two, 3 *
2^a, other and ragged sizes.
"""
import math

import numpy as np
import torch

from hymd_gb300 import adjoint as hadjoint
from hymd_gb300 import field as hfield
from hymd_gb300 import force as hforce
from hymd_gb300 import pressure as hpressure
from hymd_gb300 import systems
from hymd_gb300.config import Config
from hymd_gb300.force import Chi
from hymd_gb300.hamiltonian import get_hamiltonian
from hymd_gb300.md import RespaMD
from hymd_gb300.replicas import ReplicaBatch
from hymd_gb300.reverse import ForceModel, profile_loss

GAS = 0.0083144621
COULOMB = 138.935458
RANDOM_STEPS = 20000  # rows of the coupling's random table, as the benchmark draws
N_BINS = 100


# ------------------------------------------------------------------ cases ---
def listed():
    return [
        # the smallest simulations: every launch counts (10k-bead melt)
        dict(name="md_melt_10k", kind="md", recipe="melt", n=10000, box=10.0, nx=32, ny=32,
             nz=32, barostat=False),
        # an ordinary membrane simulation at constant pressure
        dict(name="md_membrane_162k_npt", kind="md", recipe="membrane", n=162000, box=27.0,
             nx=64, ny=64, nz=64, barostat=True),
        # the largest simulation: charged peptides, electrostatics, four-body terms
        dict(name="md_peptide_500k_pic", kind="md", recipe="peptide", n=500000, box=40.0,
             nx=128, ny=128, nz=128, barostat=False, n_res=50),
        # a parameter sweep: small systems of different sizes side by side
        dict(name="replicas_8", kind="replicas", count=8, n_min=5000, n_max=20000),
        # slow forces of a test-sized system: the smallest calls, latency and host path
        dict(name="field_melt_2k", kind="field", recipe="mixture", n=2000, types=2, box=6.2,
             nx=16, ny=16, nz=16, functional="DefaultWithChi", pic=False),
        # a box that is not a cube on a mesh with odd sizes, with charges
        dict(name="field_ragged_41k_pic", kind="field", recipe="mixture", n=41013, types=3,
             box=17.0, nx=45, ny=40, nz=54, functional="DefaultNoChi", pic=True),
        # the largest slow-force evaluation: 1.3M-bead membrane
        dict(name="field_membrane_1300k", kind="field", recipe="bilayer", n=1300000, types=5,
             box=54.0, nx=128, ny=128, nz=128, functional="DefaultWithChi", pic=False),
        # variable dielectric around charged peptides
        dict(name="gpe_peptide_61k", kind="gpe", n=61000, box=20.0, nx=64, ny=64, nz=64,
             n_res=30),
        # bonded terms of the largest peptide system through the per-term calls
        dict(name="bonded_peptide_500k", kind="bonded", recipe="peptide", n=500000, box=40.0,
             n_res=50),
        # a print step of the membrane: energies, 18-component pressure
        dict(name="report_membrane_162k", kind="report", recipe="bilayer", n=162000, types=5,
             box=27.0, nx=64, ny=64, nz=64, pic=False),
        # fitting chi to energies: gradients of the field energy of the large membrane
        dict(name="adjoint_membrane_1300k", kind="adjoint", recipe="bilayer", n=1300000,
             types=5, box=54.0, nx=128, ny=128, nz=128),
        # fitting chi to structure: a differentiated stretch of trajectory
        dict(name="reverse_membrane_40k", kind="reverse", n=40000, box=17.0, nx=48, ny=48,
             nz=48, steps=2),
    ]


FUSED = (16, 24, 32, 48, 64, 96, 128)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh(rng, box, top=128):
    """Mesh sizes at a spacing of 0.3 to 0.5 nm: a common FFT length, any
    integer, or three different ones."""
    want = min(top, max(12, box / rng.uniform(0.3, 0.5)))
    how = rng.random()
    if how < 0.5:
        m = min(FUSED, key=lambda f: abs(f - want))
        return m, m, m
    if how < 0.75:
        m = int(round(want))
        return m, m, m
    return tuple(max(12, min(top, int(round(want * rng.uniform(0.85, 1.15))))) for _ in range(3))


def draw(rng):
    kind = rng.choice(["md", "md", "md", "md", "replicas", "field", "field", "field", "gpe",
                       "bonded", "report", "adjoint", "reverse"])
    density = rng.uniform(7.5, 10.0)
    if kind == "replicas":
        lo = _log_int(rng, 2000, 8000)
        return dict(kind=kind, count=rng.randint(3, 8), n_min=lo,
                    n_max=_log_int(rng, lo + 500, 20000))
    if kind in ("md", "bonded"):
        recipe = rng.choice(["melt", "membrane", "peptide"])
        n = _log_int(rng, 2000 if recipe == "melt" else 6000, 500000)
        box = round((n / density) ** (1 / 3), 3)
        case = dict(kind=kind, recipe=recipe, n=n, box=box)
        if recipe == "peptide":
            case["n_res"] = rng.randint(8, 50)
        if kind == "md":
            case["nx"], case["ny"], case["nz"] = _mesh(rng, box)
            case["barostat"] = recipe != "peptide" and rng.random() < 0.4
        return case
    if kind == "gpe":
        n = _log_int(rng, 5000, 300000)
        box = round((n / density) ** (1 / 3), 3)
        nx, ny, nz = _mesh(rng, box)
        return dict(kind=kind, n=n, box=box, nx=nx, ny=ny, nz=nz, n_res=rng.randint(8, 50))
    if kind == "reverse":
        n = _log_int(rng, 5000, 40000)
        box = round((n / density) ** (1 / 3), 3)
        nx, ny, nz = _mesh(rng, box)
        return dict(kind=kind, n=n, box=box, nx=nx, ny=ny, nz=nz, steps=rng.randint(1, 2))
    bilayer = rng.random() < 0.5
    n = _log_int(rng, 5000 if bilayer else 2000, 1300000)
    box = round((n / density) ** (1 / 3), 3)
    nx, ny, nz = _mesh(rng, box)
    case = dict(kind=kind, recipe="bilayer" if bilayer else "mixture", n=n,
                types=5 if bilayer else rng.randint(1, 5), box=box, nx=nx, ny=ny, nz=nz)
    if kind == "field":
        case["functional"] = rng.choice(["DefaultWithChi", "DefaultNoChi", "SquaredPhi"])
    if kind != "adjoint":
        case["pic"] = rng.random() < 0.4
    return case


# ---------------------------------------------------------------- systems ---
def _built(case, seed):
    """A system of the repository's recipes with topology, on the host."""
    n, box = case["n"], case["box"]
    mesh = [case.get("nx", 32), case.get("ny", 32), case.get("nz", 32)]
    recipe = case.get("recipe", "peptide" if case["kind"] == "gpe" else "membrane")
    if recipe == "melt":
        s = systems.homopolymer_melt(seed=seed, n_chains=n // 10, length=10, box=box, mesh=mesh)
    elif recipe == "membrane":
        lipids = int(0.444 * n / 12)
        s = systems.lipid_membrane(seed=seed, n_lipids=lipids, n_water=n - 12 * lipids, box=box,
                                   mesh=mesh)
    else:
        per = 2 * case["n_res"]
        s = systems.charged_peptides(seed=seed, n_chains=max(1, n // 25 // per),
                                     n_res=case["n_res"], n_total=n, box=box, mesh=mesh)
    if recipe != "membrane":
        # the random walks place bonded beads exactly at the bonds' rest
        # lengths: a thermal displacement as in a running simulation
        rng = np.random.default_rng(seed + 1)
        r = s["positions"] + rng.normal(0.0, 0.03, s["positions"].shape)
        s["positions"] = np.mod(r, s["config"].box()).astype(np.float32)
    cfg = s["config"]
    if not case.get("barostat", False):
        cfg.barostat = None
    elif cfg.barostat is None:
        cfg.barostat, cfg.tau_p, cfg.n_b = "isotropic", 1.0, 1
        cfg.rho0 = cfg.a = cfg.n_particles / float(np.prod(cfg.box()))
    return s


def _sweep(case, seed):
    """Melts and membranes in turn, their sizes spread between the case's
    limits, chi different in each."""
    out = []
    for i in range(case["count"]):
        f = i / max(1, case["count"] - 1)
        n = int(case["n_min"] ** (1 - f) * case["n_max"] ** f) // 10 * 10
        box = round((n / 8.3) ** (1 / 3), 3)
        mesh = min(systems.REPLICA_MESHES, key=lambda m: abs(m - box / 0.4))
        chi = 5.0 + 5.0 * i
        if i % 2 == 0:
            s = systems.homopolymer_melt(seed=seed + i, n_chains=n // 10, box=box, mesh=mesh,
                                         chi_ab=chi)
        else:
            lipids = int(0.444 * n / 12)
            s = systems.lipid_membrane(seed=seed + i, n_lipids=lipids, n_water=n - 12 * lipids,
                                       box=box, mesh=mesh, chi_cw=chi)
        s["config"].barostat = None
        out.append(s)
    return out


def _beads(case, seed):
    """Positions, velocities, types, charges of a mixture (uniform, some of
    it clustered) or a bilayer in water, made on the GPU, and its Config."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, T, L = case["n"], case["types"], case["box"]
    rand = lambda *s: torch.rand(*s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    if case["recipe"] == "bilayer":
        box = np.full(3, L)
        lip = int(0.444 * n / 12)
        # N P G G and two tails of four C; types in name order C G N P W
        kinds = torch.tensor([2, 3, 1, 1, 0, 0, 0, 0, 0, 0, 0, 0], device="cuda")
        depth = torch.tensor([0, 1, 2, 2, 3, 4, 5, 6, 3, 4, 5, 6], device="cuda").double()
        xy = rand(lip, 1, 2) * L
        up = torch.where(torch.arange(lip, device="cuda") % 2 == 0, 1.0, -1.0).double()[:, None]
        z = L / 2 + up * (2.0 - 0.26 * depth)
        pos = torch.cat([xy.expand(lip, 12, 2), z[:, :, None]], 2) + 0.15 * randn(lip, 12, 3)
        w = rand(n - 12 * lip, 3) * L
        slab = min(2.6, 0.3 * L)
        w[:, 2] = L / 2 + slab + w[:, 2] * (1 - 2 * slab / L)
        r = torch.cat([pos.reshape(-1, 3), w])
        types = torch.cat([kinds.repeat(lip), torch.full((n - 12 * lip,), 4, device="cuda")])
    else:
        box = np.array([L, 0.9 * L, 1.1 * L])
        r = rand(n, 3) * torch.tensor(box, device="cuda")
        k = n // 4
        r[:k] = 0.5 * torch.tensor(box, device="cuda") + 0.15 * L * randn(k, 3)
        types = torch.randint(0, T, (n,), generator=g, device="cuda")
    Lt = torch.tensor(box, device="cuda")
    r = torch.remainder(r, Lt).float()
    r = torch.where(r >= Lt.float(), torch.zeros_like(r), r).contiguous()
    v = (randn(n, 3) * math.sqrt(GAS * 323.0 / 72.0)).float().contiguous()
    q = None
    if case.get("pic"):
        u = rand(n)
        q = torch.where(u < 0.1, 1.0, torch.where(u < 0.2, -1.0, 0.0)).float().contiguous()
    names = ["C", "G", "N", "P", "W"][:T]
    chi = [Chi(names[i], names[j], 4.0 + 3.0 * i + 5.0 * (j - i)) for i in range(T)
           for j in range(i + 1, T)]
    cfg = Config(n_steps=1, time_step=0.03, mesh_size=[case["nx"], case["ny"], case["nz"]],
                 sigma=0.5, kappa=0.05, box_size=box, n_particles=n, n_types=T, mass=72.0,
                 hamiltonian=case.get("functional", "DefaultWithChi"), unique_names=names,
                 type_to_name_map=dict(enumerate(names)), chi=chi, m=[1.0] * T,
                 coulombtype="PIC_Spectral" if q is not None else None, dielectric_const=15.0,
                 type_charges=[0.25 * (-1) ** t for t in range(T)])
    return r, v, types.int().contiguous(), q, cfg


def _chi_matrix(cfg):
    T = cfg.n_types
    idx = {n: i for i, n in enumerate(cfg.unique_names)}
    chi = np.zeros((T, T))
    for c in cfg.chi:
        i, j = idx[c.atom_1], idx[c.atom_2]
        chi[i, j] = chi[j, i] = c.interaction_energy
    return chi


def _simulation(s, seed, barostat):
    cfg = s["config"]
    md = RespaMD(s["positions"], s["velocities"], s["types"], cfg, get_hamiltonian(cfg),
                 topology=s["topology"], charges=s.get("charges"))
    md.sort_particles()
    md.couple(thermostat=True, barostat="isotropic" if barostat else None, seed=seed,
              n_steps=RANDOM_STEPS)
    md.prime()
    md.capture()
    return md


def _mesh_objects(cfg):
    pm, fields, elec, coulomb = hfield.initialize_pm(None, cfg)
    return dict(pm=pm, fields=fields, elec=elec, coulomb=coulomb)


def _slow_density(st):
    phi, phi_fourier, fmesh, v_ext_fourier, v_ext, phi_transfer, phi_lap = st["fields"]
    hfield.update_field(phi, phi_lap, phi_transfer, None, fmesh, st["ham"], st["pm"], st["r"],
                        st["types"], st["cfg"], v_ext, phi_fourier, v_ext_fourier, st["cfg"].m)


def _slow_charge(st):
    phi_q, phi_q_fourier, psi, elec_field = st["elec"]
    elec_field_fourier, psi_fourier = st["coulomb"]
    hfield.update_field_force_q(st["q"], phi_q, phi_q_fourier, psi, psi_fourier,
                                elec_field_fourier, elec_field, st["f_elec"], None, st["ham"],
                                st["pm"], st["r"], st["cfg"])


# ---------------------------------------------------------------- prepare ---
def prepare(case, seed):
    kind = case["kind"]
    if kind == "md":
        md = _simulation(_built(case, seed), seed, case["barostat"])
        return dict(kind=kind, md=md, barostat=case["barostat"])
    if kind == "replicas":
        batch = ReplicaBatch(_sweep(case, seed), seed=seed, n_steps=RANDOM_STEPS)
        batch.prime()
        batch.capture(n_streams=8)
        return dict(kind=kind, batch=batch)
    if kind == "bonded":
        s = _built(case, seed)
        n = len(s["positions"])
        real = {2, 3, 7, 8, 13}
        topo = [torch.as_tensor(np.asarray(x, np.float32 if i in real else np.int32),
                                device="cuda") for i, x in enumerate(s["topology"])]
        nd = topo[9].numel()
        z = lambda *d: torch.zeros(*d, dtype=torch.float32, device="cuda")  # noqa: E731
        return dict(kind=kind, r=torch.as_tensor(s["positions"], device="cuda"), topo=topo,
                    box=torch.as_tensor(s["config"].box(), device="cuda"),
                    f=[z(n, 3) for _ in range(3)], dipoles=z(nd, 4, 3), transfer=z(nd, 6, 3, 3))
    if kind == "gpe":
        s = _built(case, seed)
        cfg = _gpe_config(s["config"])
        st = dict(kind=kind, cfg=cfg, ham=get_hamiltonian(cfg),
                  r=torch.as_tensor(s["positions"], device="cuda"),
                  types=torch.as_tensor(s["types"], device="cuda"),
                  q=torch.as_tensor(s["charges"], device="cuda"), **_mesh_objects(cfg))
        _slow_density(st)
        st["f_elec"] = torch.zeros_like(st["r"])
        return st
    if kind == "reverse":
        s = _built(case, seed)
        cfg = s["config"]
        md = RespaMD(s["positions"], s["velocities"], s["types"], cfg, get_hamiltonian(cfg),
                     topology=s["topology"])
        chi = torch.tensor(_chi_matrix(cfg), dtype=torch.float32, device="cuda",
                           requires_grad=True)
        x = md.r.clone().requires_grad_(True)
        v = md.v.clone().requires_grad_(True)
        return dict(kind=kind, md=md, model=ForceModel(md), x=x, v=v, chi=chi,
                    steps=case["steps"], target=_target(case, cfg, seed).float())
    r, v, types, q, cfg = _beads(case, seed)
    ham = get_hamiltonian(cfg)
    if kind == "adjoint":
        chi = torch.tensor(_chi_matrix(cfg), dtype=torch.float32, device="cuda",
                           requires_grad=True)
        pm = hfield.ParticleMesh(cfg.mesh_size, cfg.box_size, cfg.n_types)
        return dict(kind=kind, r=r.requires_grad_(True), types=types, chi=chi, pm=pm, cfg=cfg)
    st = dict(kind=kind, r=r, v=v, types=types, q=q, cfg=cfg, ham=ham,
              force=torch.zeros_like(r), f_elec=torch.zeros_like(r), **_mesh_objects(cfg))
    if kind == "report":
        _slow_density(st)
        if q is not None:
            cfg.self_energy = hfield.compute_self_energy_q(cfg, q)
            _slow_charge(st)
        st["bond_pr"], st["angle_pr"] = _virials(case, seed)
    return st


def _gpe_config(cfg):
    cfg.coulombtype = "PIC_Spectral_GPE"
    cfg.dielectric_type = [2.0, 10.0, 80.0]
    cfg.conv_crit, cfg.pol_mixing, cfg.convergence_type = 1e-6, 0.6, "max_diff"
    cfg.type_charges = [0.05, -0.05, 0.0]
    return cfg


def _virials(case, seed):
    rng = np.random.default_rng(seed)
    scale = 10.0 * case["n"]
    return rng.normal(0, scale, 3).astype(np.float32), rng.normal(0, scale, 3).astype(np.float32)


def _target(case, cfg, seed):
    """A smooth profile to fit: per type, its mean density with a cosine."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    z = (torch.arange(N_BINS, device="cuda").double() + 0.5) / N_BINS
    amp = torch.rand(cfg.n_types, 2, generator=g, device="cuda", dtype=torch.float64)
    rho = cfg.n_particles / float(np.prod(cfg.box())) / cfg.n_types
    return rho * (1.0 + 0.5 * amp[:, :1] * torch.cos(2 * math.pi * (z[None] + amp[:, 1:])))


# -------------------------------------------------------------------- run ---
def run(state):
    kind = state["kind"]
    if kind == "md":
        md = state["md"]
        md.run(1)
        out = dict(r=md.r, v=md.v, f_field=md.f_field, f_bonded=md.f_b)
        if md.f_elec is not None:
            out["f_elec"] = md.f_elec
        if state["barostat"]:
            out["box"] = md.box.clone()  # (md.box is a view of the mesh's own state)
        return out
    if kind == "replicas":
        state["batch"].run(1)
        return [dict(r=md.r, v=md.v, f_field=md.f_field) for md in state["batch"].replicas]
    if kind == "field":
        _slow_density(state)
        phi, phi_fourier, fmesh = state["fields"][:3]
        hfield.compute_field_force(None, state["r"], fmesh, state["force"], state["types"],
                                   state["cfg"].n_types)
        out = dict(phi=phi, phi_fourier=phi_fourier, mesh=fmesh, force=state["force"])
        if state["q"] is not None:
            _slow_charge(state)
            phi_q, _, psi, elec_field = state["elec"]
            out.update(phi_q=phi_q, psi=psi, elec_field=elec_field, f_elec=state["f_elec"],
                       psi_fourier=state["coulomb"][1])
        return out
    if kind == "gpe":
        phi = state["fields"][0]
        phi_q, phi_q_fourier, psi, elec_field = state["elec"]
        (eps, eps_fourier, eta, eta_fourier, pol, pol_prev, _, contrib, vbar, vbar_fourier, fme,
         fme_fourier) = state["coulomb"]
        vbar, eps, dot = hfield.update_field_force_q_GPE(
            None, phi, state["types"], state["q"], phi_q, phi_q_fourier, eps, eps_fourier, eta,
            eta_fourier, pol_prev, pol, elec_field, state["f_elec"], contrib, psi, vbar,
            vbar_fourier, fme, fme_fourier, state["ham"], None, None, state["pm"], state["r"],
            state["cfg"])
        return dict(vbar=vbar, eps=eps, dot=dot, psi=psi, elec_field=elec_field,
                    f_elec=state["f_elec"])
    if kind == "bonded":
        (b2a, b2b, b2r, b2k, b3a, b3b, b3c, b3t, b3k, b4a, b4b, b4c, b4d, coeff, dtype,
         last) = state["topo"]
        fb, fa, fd = state["f"]
        r, box = state["r"], state["box"]
        eb, pb = hforce.compute_bond_forces(fb, r, box, b2a, b2b, b2r, b2k)
        out = dict(e_bond=eb, pr_bond=pb, f_bond=fb)
        if b3a.numel():
            ea, pa = hforce.compute_angle_forces(fa, r, box, b3a, b3b, b3c, b3t, b3k)
            out.update(e_angle=ea, pr_angle=pa, f_angle=fa)
        if b4a.numel():
            ed = hforce.compute_dihedral_forces(fd, r, state["dipoles"], state["transfer"], box,
                                                b4a, b4b, b4c, b4d, coeff, dtype, last, 1)
            out.update(e_dihedral=ed, f_dihedral=fd, dipoles=state["dipoles"],
                       transfer=state["transfer"])
        return out
    if kind == "report":
        phi, phi_fourier, _, _, v_ext, phi_transfer, phi_lap = state["fields"]
        phi_q, _, psi, _ = state["elec"]
        w, ke, wq = hfield.compute_field_and_kinetic_energy(
            phi, phi_q, psi, state["v"], state["ham"], state["r"], state["types"], v_ext,
            state["cfg"], None)
        p = hpressure.comp_pressure(phi, phi_q, psi, state["ham"], state["v"], state["cfg"],
                                    phi_fourier, phi_lap, phi_transfer, state["r"],
                                    state["bond_pr"], state["angle_pr"])
        return dict(w=w, ke=ke, wq=wq, pressure=p, laplacian=phi_lap)
    if kind == "adjoint":
        cfg = state["cfg"]
        w = hadjoint.field_energy(state["r"], state["types"], state["pm"], cfg.m, state["chi"],
                                  cfg.kappa, cfg.sigma, cfg.rho0, cfg.a)
        gx, gchi = torch.autograd.grad(w, [state["r"], state["chi"]])
        return dict(w=w, dx=gx, dchi=gchi)
    x, v, chi = state["x"], state["v"], state["chi"]
    loss, prof = profile_loss(x, v, chi, state["model"], state["steps"], state["target"], N_BINS)
    gx, gv, gchi = torch.autograd.grad(loss, [x, v, chi])
    return dict(loss=loss, profile=prof, dx=gx, dv=gv, dchi=gchi)


# ------------------------------------------------------------------- work ---
def work(case):
    """Inputs read once and outputs written once; transforms at 2.5 M log2 M
    per real grid, about 30 operations per bead and grid for deposits and
    gathers, and per bonded term."""
    kind = case["kind"]
    if kind == "replicas":
        n = case["count"] * math.sqrt(case["n_min"] * case["n_max"])
        M = n / 8.3 / 0.4 ** 3
        return dict(bytes=100.0 * n, flops=1000.0 * n + 8 * 2.5 * M * math.log2(32 ** 3))
    n = case["n"]
    T = {"melt": 2, "membrane": 5, "peptide": 3}.get(case.get("recipe"), case.get("types", 5))
    if kind == "gpe":
        T = 3
    lip = 0.444 * n
    terms = {"melt": 0.9 * n, "membrane": 2.2 * lip, "peptide": 0.1 * n}.get(
        case.get("recipe"), 2.2 * lip)
    if kind == "bonded":
        return dict(bytes=12.0 * n * (2 + 2 * (case["recipe"] != "melt")) + 24.0 * terms,
                    flops=80.0 * terms)
    M = float(case["nx"] * case["ny"] * case["nz"])
    fft = 2.5 * M * math.log2(M)
    if kind == "md":
        q = case["recipe"] == "peptide"
        return dict(bytes=n * (2 * (24 + 24 + 12 * q) + 4 + 4 * q),
                    flops=(4 * T + 4 * q) * fft + 30 * n * (2 + q) + 10 * (80 * terms + 12 * n))
    if kind == "field":
        q = bool(case["pic"])
        grids = T * 20 * M + q * 24 * M  # densities, spectra, force mesh; charge grids
        return dict(bytes=16.0 * n + 12 * n + q * 16 * n + grids,
                    flops=(5 * T + 5 * q) * fft + 60.0 * n)
    if kind == "gpe":
        return dict(bytes=32.0 * n + 4 * M * (2 * T + 8), flops=(4 * T + 40) * fft)
    if kind == "report":
        return dict(bytes=28.0 * n + 4 * M * T * 4, flops=(T + 3 * T) * fft)
    if kind == "adjoint":
        return dict(bytes=28.0 * n, flops=2 * T * fft + 60.0 * n)
    steps = case["steps"]
    return dict(bytes=60.0 * n, flops=steps * (12 * T * fft + 600 * terms + 200.0 * n))


# ------------------------------------------------------------------ exact ---
# The same quantities in 64 bits: plain torch in double precision.
class _Mesh64:
    def __init__(self, mesh, box, sigma):
        self.n = tuple(int(x) for x in mesh)
        self.box = torch.as_tensor(box, dtype=torch.float64, device="cuda").reshape(3)
        self.M = self.n[0] * self.n[1] * self.n[2]
        self.V = float(self.box.prod())
        self.dV = self.V / self.M
        L = [float(x) for x in self.box]
        ks = [2 * math.pi / L[d] * torch.fft.fftfreq(self.n[d], 1.0 / self.n[d],
                                                     dtype=torch.float64, device="cuda")
              for d in range(2)]
        ks.append(2 * math.pi / L[2] * torch.arange(self.n[2] // 2 + 1, device="cuda").double())
        shapes = [(-1, 1, 1), (1, -1, 1), (1, 1, -1)]
        self.k = [k.reshape(s) for k, s in zip(ks, shapes)]
        self.g = []
        for d, k in enumerate(self.k):
            k = k.clone()
            if self.n[d] % 2 == 0:
                k.reshape(-1)[self.n[d] // 2] = 0.0
            self.g.append(k)
        self.k2 = self.k[0] ** 2 + self.k[1] ** 2 + self.k[2] ** 2
        self.H = torch.exp(-0.5 * sigma * sigma * self.k2)
        self.kn = self.k2.clone()
        self.kn[0, 0, 0] = 1.0
        w = torch.full((self.n[2] // 2 + 1,), 2.0, dtype=torch.float64, device="cuda")
        w[0] = 1.0
        if self.n[2] % 2 == 0:
            w[-1] = 1.0
        self.w = w  # multiplicity of the half spectrum

    def r2c(self, f):
        return torch.fft.rfftn(f, dim=(-3, -2, -1)) / self.M

    def c2r(self, f):
        return torch.fft.irfftn(f * self.M, s=self.n, dim=(-3, -2, -1))

    def cic(self, r):
        """Flat corner indices and weights, (8, N)."""
        s = r / self.box * torch.tensor(self.n, device="cuda", dtype=torch.float64)
        i0 = torch.floor(s).detach()
        f = s - i0
        i0 = i0.long()
        idx, w = [], []
        for a in (0, 1):
            for b in (0, 1):
                for c in (0, 1):
                    i = [(i0[:, d] + o) % self.n[d] for d, o in enumerate((a, b, c))]
                    idx.append((i[0] * self.n[1] + i[1]) * self.n[2] + i[2])
                    wd = [f[:, d] if o else 1.0 - f[:, d] for d, o in enumerate((a, b, c))]
                    w.append(wd[0] * wd[1] * wd[2])
        return torch.stack(idx), torch.stack(w)

    def paint(self, cic, slot, weight, slots):
        idx, w = cic
        flat = torch.zeros(slots * self.M, dtype=torch.float64, device="cuda")
        at = (slot[None, :] * self.M + idx).reshape(-1)
        return flat.index_add(0, at, (w * weight[None, :]).reshape(-1)).reshape(slots, *self.n)

    def readout(self, cic, grids, slot):
        """grids (S, 3, mesh) at each bead's slot: (N, 3)."""
        idx, w = cic
        flat = grids.reshape(-1)
        cols = [(w * flat[(slot[None, :] * 3 + d) * self.M + idx]).sum(0) for d in range(3)]
        return torch.stack(cols, 1)

    def gradient(self, spec):
        """c2r(-i k_d spec) for d = 0, 1, 2 on a new axis before the mesh."""
        return torch.stack([self.c2r(-1j * g * spec) for g in self.g], dim=-4)


def _functional(cfg, kind=None):
    """(Q, b, c) of w = 1/2 phi.Q.phi + b.phi + c."""
    kind = kind or cfg.hamiltonian
    T = cfg.n_types
    rho0 = cfg.n_particles / float(np.prod(np.asarray(cfg.box_size, dtype=np.float64)))
    inc = 1.0 / (cfg.kappa * rho0)
    Q = np.full((T, T), inc)
    if kind == "DefaultWithChi":
        Q = Q + _chi_matrix(cfg) / rho0
    a = 0.0 if kind == "SquaredPhi" else rho0
    return torch.tensor(Q, device="cuda"), -a * inc, 0.5 * a * a * inc


def _field64(m, r, types, T, Q, b):
    t = types.long()
    cic = m.cic(r)
    phi_raw = m.paint(cic, t, torch.ones_like(r[:, 0]) / m.dV, T)
    spec = m.r2c(phi_raw) * m.H
    v = torch.einsum("tj,jxyz->txyz", Q.to(spec.dtype), spec)
    v[:, 0, 0, 0] += b
    mesh = m.gradient(v * m.H)
    return dict(cic=cic, spec=spec, mesh=mesh, force=m.readout(cic, mesh, t))


def _pic64(m, r, q, factor, cic):
    zero = torch.zeros_like(cic[0][0])
    phi_q = m.paint(cic, zero, q / m.dV, 1)
    psi_k = 4 * math.pi * factor * m.r2c(phi_q) * m.H / m.kn
    E = m.gradient(psi_k)
    return dict(phi_q=phi_q[0], psi_k=psi_k[0], psi=m.c2r(psi_k)[0], E=E[0],
                force=q[:, None] * m.readout(cic, E, zero))


def _image(d, box):
    return d - box * torch.round(d / box)


def _bond64(x, box, topo):
    a, b, r0, k = topo[0], topo[1], topo[2], topo[3]
    rab = _image(x[b] - x[a], box)
    d = torch.linalg.norm(rab, dim=1)
    f = (-k * (d - r0) / d)[:, None] * rab
    return 0.5 * (k * (d - r0) ** 2).sum(), (f.detach() * rab.detach()).sum(0)


def _angle64(x, box, topo):
    a, b, c, t0, k = topo[4], topo[5], topo[6], topo[7], topo[8]
    ra, rc = _image(x[a] - x[b], box), _image(x[c] - x[b], box)
    na, nc = torch.linalg.norm(ra, dim=1), torch.linalg.norm(rc, dim=1)
    ea, ec = ra / na[:, None], rc / nc[:, None]
    s, co = torch.linalg.norm(torch.linalg.cross(ea, ec), dim=1), (ea * ec).sum(1)
    d = torch.atan2(s, co) - t0
    with torch.no_grad():
        ga = (-k * d / (na * s))[:, None] * (ec - co[:, None] * ea)
        gc = (-k * d / (nc * s))[:, None] * (ea - co[:, None] * ec)
        vir = -(ga * ra + gc * rc).sum(0)
    return 0.5 * (k * d * d).sum(), vir


def _series(c, d, phi):
    n = torch.arange(5, dtype=torch.float64, device="cuda")
    return (c * (1.0 + torch.cos(n * phi[:, None] - d))).sum(1)


def _dihedral64(x, box, topo):
    """Cosine series, combined bending-torsion and improper terms.  The
    gradient of the bending angle keeps the reference's lower limit of 0.1
    on its sine."""
    a, b, c, d, cf, ty, last = topo[9:16]
    f, g, h = _image(x[a] - x[b], box), _image(x[b] - x[c], box), _image(x[d] - x[c], box)
    v, w = torch.linalg.cross(f, g), torch.linalg.cross(h, g)
    phi = torch.atan2((w * f).sum(1) * torch.linalg.norm(g, dim=1), (v * w).sum(1))
    e = _series(cf[:, 0], cf[:, 1], phi)
    both = (cf[:, 2] != 0).any(1) & (cf[:, 3] != 0).any(1)
    e = e + torch.where(both, _series(cf[:, 2], cf[:, 3], phi), 0.0)
    e = e * ((ty == 0) | (ty == 1)).double()
    K = _series(cf[:, 4], cf[:, 5], phi)
    gamma0 = 1.85 - 0.227 * torch.cos(phi - float(np.float32(0.785)))

    def bend(p, q):
        cg = (p * q).sum(1) / (torch.linalg.norm(p, dim=1) * torch.linalg.norm(q, dim=1))
        c0 = cg.detach()
        slope = -1.0 / torch.sqrt(1.0 - c0 * c0).clamp_min(0.1)
        gamma = torch.acos(c0) + slope * (cg - c0)
        return 0.5 * K * (gamma - gamma0) ** 2

    cbt = (ty == 1).double()
    e = e + bend(f, -g) * cbt + bend(g, h) * cbt * (last == 1).double()
    imp = 0.5 * cf[:, 0, 1] * (phi - cf[:, 0, 0]) ** 2
    return (e + imp * (ty == 2).double()).sum()


def _topo64(topo):
    """Indices as they are, parameters as the float32 values kernels take."""
    real = {2, 3, 7, 8, 13}
    out = []
    for i, x in enumerate(topo):
        x = torch.as_tensor(np.asarray(x), device="cuda")
        out.append(x.float().double() if i in real else x.long())
    out[13] = out[13].reshape(-1, 6, 5)
    return out


def _bonded64(x, box, topo, graph=False):
    """(force, bond virial, angle virial) of all bonded terms."""
    if not x.requires_grad:
        x = x.detach().requires_grad_(True)
    zero = torch.zeros(3, dtype=torch.float64, device="cuda")
    e, vb, va = 0.0, zero, zero
    if len(topo[0]):
        eb, vb = _bond64(x, box, topo)
        e = e + eb
    if len(topo[4]):
        ea, va = _angle64(x, box, topo)
        e = e + ea
    if len(topo[9]):
        e = e + _dihedral64(x, box, topo)
    return -torch.autograd.grad(e, x, create_graph=graph)[0], vb, va


def _cell_order(s, r, mesh, box):
    """The stable bead order of `sort_particles`: by the mesh cell of each
    molecule's first bead, then by that bead."""
    n = len(r)
    lab = torch.arange(n, device="cuda")
    topo = s["topology"]
    pairs = [(0, 1), (4, 5), (5, 6), (9, 10), (10, 11), (11, 12)]
    pairs = [(torch.as_tensor(np.asarray(topo[i], np.int64), device="cuda"),
              torch.as_tensor(np.asarray(topo[j], np.int64), device="cuda")) for i, j in pairs]
    a, b = (torch.cat([p[k] for p in pairs]) for k in (0, 1))
    while len(a):
        low = torch.minimum(lab[a], lab[b])
        new = lab.clone()
        new.scatter_reduce_(0, a, low, "amin")
        new.scatter_reduce_(0, b, low, "amin")
        new = new[new]
        if torch.equal(new, lab):
            break
        lab = new
    nn = torch.tensor(mesh, dtype=torch.float64, device="cuda")
    c = torch.remainder(torch.floor(r / box * nn).long(), nn.long())
    key = (c[:, 0] * mesh[1] + c[:, 1]) * mesh[2] + c[:, 2]
    return torch.argsort(key[lab] * n + lab, stable=True)


def _md64(s, seed, barostat, steps):
    """`steps` outer rRESPA steps from the initial state, in the memory order
    that the simulation keeps."""
    cfg = s["config"]
    mesh = tuple(int(x) for x in cfg.mesh())
    r = torch.as_tensor(s["positions"], device="cuda").double()
    v = torch.as_tensor(s["velocities"], device="cuda").double()
    types = torch.as_tensor(s["types"], device="cuda")
    q = s.get("charges")
    q = None if q is None else torch.as_tensor(q, device="cuda").double()
    topo = _topo64(s["topology"])
    box = torch.as_tensor(cfg.box(), device="cuda")
    perm = _cell_order(s, r, mesh, box)
    N, T, mass, dt, inner = len(r), cfg.n_types, float(cfg.mass), cfg.time_step, cfg.respa_inner
    Q, b, c = _functional(cfg)
    dto = inner * dt
    rng = np.random.default_rng(seed)

    def slow(r, box):
        m = _Mesh64(mesh, box, cfg.sigma)
        f = _field64(m, r, types, T, Q, b)
        fq = None
        if q is not None:
            fq = _pic64(m, r, q, COULOMB / cfg.dielectric_const, f["cic"])["force"]
        sums = None
        if barostat:
            p = f["spec"]
            e = torch.einsum("txyz,tj,jxyz->xyz", p.conj(), Q.to(p.dtype), p).real * m.w
            e[0, 0, 0] = 0.0
            sums = [float(e.sum())] + [float((e * k * k).sum()) for k in m.k]
        return f["force"], fq, sums

    ff, fq, sums = slow(r, box)
    fb, vb, va = _bonded64(r, box, topo)
    for _ in range(steps):
        kick = ff if fq is None else ff + fq
        v = v + 0.5 * dto * kick / mass
        for _ in range(inner):
            v = v + 0.5 * dt * fb / mass
            r = torch.remainder(r + dt * v, box)
            fb, vb, va = _bonded64(r, box, topo)
            v = v + 0.5 * dt * fb / mass
        if barostat:
            V = float(box.prod())
            counts = torch.bincount(types.long(), minlength=T).double()
            p01 = 0.5 * sums[0] + 0.5 * float(counts @ Q @ counts) / V ** 2 - c
            kin = mass * float((v * v).sum()) / (3.0 * V)
            p = [kin + p01 - cfg.sigma ** 2 * sums[1 + d] + float(vb[d] + va[d]) / V
                 for d in range(2)]
            P = 0.5 * (p[0] + p[1]) * 16.61
            beta, tau, nb = 7.6e-4, cfg.tau_p, float(cfg.n_b)
            kT = cfg.gas_constant * cfg.target_temperature
            noise = math.sqrt(2.0 * nb * kT * beta * dto * nb / (V * tau)) * rng.normal()
            alpha = math.exp((-nb * dto * beta / tau * (1.0 - P) + noise) / 3.0)
            box, r = box * alpha, r * alpha
        ff, fq, sums = slow(r, box)
        v = v + 0.5 * dto * (ff if fq is None else ff + fq) / mass
        R, S = rng.normal(), rng.chisquare(3 * N - 1)
        com = v.mean(0)
        K = 0.5 * mass * float(((v - com) ** 2).sum())
        Kt = 1.5 * cfg.gas_constant * N * cfg.target_temperature
        cc = math.exp(-dto / cfg.tau)
        ratio = Kt / (3 * N * K)
        a2 = cc + (1 - cc) * (S + R * R) * ratio + 2 * R * math.sqrt(cc * (1 - cc) * ratio)
        v = (v - com) * math.sqrt(a2) + com
    out = dict(r=r[perm], v=v[perm], f_field=ff[perm], f_bonded=fb[perm])
    if fq is not None:
        out["f_elec"] = fq[perm]
    if barostat:
        out["box"] = box
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "md":
        # one step when the simulation was captured, one in run()
        return _md64(_built(case, seed), seed, case["barostat"], 2)
    if kind == "replicas":
        out = []
        for i, s in enumerate(_sweep(case, seed)):
            o = _md64(s, seed + i, False, 2)
            out.append(dict(r=o["r"], v=o["v"], f_field=o["f_field"]))
        return out
    if kind == "bonded":
        return _exact_bonded(case, seed)
    if kind == "gpe":
        return _exact_gpe(case, seed)
    if kind == "reverse":
        return _exact_reverse(case, seed)
    r, v, types, q, cfg = _beads(case, seed)
    r, T = r.double(), cfg.n_types
    m = _Mesh64(cfg.mesh(), cfg.box_size, cfg.sigma)
    if kind == "adjoint":
        return _exact_adjoint(m, r, types, cfg)
    Q, b, c = _functional(cfg)
    f = _field64(m, r, types, T, Q, b)
    spec = f["spec"]
    pic = None
    if q is not None:
        q = q.double()
        pic = _pic64(m, r, q, COULOMB / cfg.dielectric_const, f["cic"])
    if kind == "field":
        out = dict(phi=list(m.c2r(spec)), phi_fourier=list(spec),
                   mesh=[list(x) for x in f["mesh"]], force=f["force"])
        if pic is not None:
            out.update(phi_q=pic["phi_q"], psi=pic["psi"], elec_field=list(pic["E"]),
                       f_elec=pic["force"], psi_fourier=pic["psi_k"])
        return out
    # energies and pressure
    phi = m.c2r(spec)
    vext = torch.einsum("tj,jxyz->txyz", Q, phi) + b
    w = float((0.5 * (phi * (vext + b)).sum(0) + c).sum()) * m.dV
    ke = 0.5 * cfg.mass * float((v.double() ** 2).sum())
    lap = torch.stack([m.c2r(-k * k * spec) for k in m.k], dim=1)
    wq = 0.0
    if pic is not None:
        pref = COULOMB / cfg.dielectric_const * math.sqrt(1.0 / (2 * math.pi * cfg.sigma ** 2))
        wq = 0.5 * float((pic["phi_q"] * pic["psi"]).sum()) * m.dV - pref * float((q * q).sum())
        tq = torch.tensor(cfg.type_charges, device="cuda", dtype=torch.float64)
        vext = vext + tq[:, None, None, None] * pic["psi"]
    pr = [x.astype(np.float64) / m.V for x in _virials(case, seed)]
    kin, p0 = 2.0 / (3.0 * m.V) * ke, -(w + wq) / m.V
    p1 = float((vext * phi).sum()) / m.M
    p2 = np.array([cfg.sigma ** 2 * float((vext * lap[:, d]).sum()) / m.M for d in range(3)])
    total = kin + p0 + p1 + p2 + pr[0] + pr[1]
    return dict(w=w, ke=ke, wq=wq, laplacian=[list(x) for x in lap],
                pressure=np.array([kin, p0, p1, *p2, *pr[0], *pr[1], 0, 0, 0, *total]))


def _exact_adjoint(m, r, types, cfg):
    T = cfg.n_types
    x = r.requires_grad_(True)
    chi = torch.tensor(_chi_matrix(cfg), device="cuda", requires_grad=True)
    rho0 = cfg.n_particles / m.V
    inc = 1.0 / (cfg.kappa * rho0)
    Q = inc + 0.5 * (chi + chi.T) * (1 - torch.eye(T, device="cuda").double()) / rho0
    phi = m.paint(m.cic(x), types.long(), torch.ones_like(x[:, 0]) / m.dV, T)
    phi = m.c2r(m.r2c(phi) * m.H)
    quad = 0.5 * (phi * torch.einsum("tj,jxyz->txyz", Q, phi)).sum()
    w = (quad - rho0 * inc * phi.sum() + 0.5 * rho0 * rho0 * inc * m.M) * m.dV
    gx, gchi = torch.autograd.grad(w, [x, chi])
    return dict(w=w.detach(), dx=gx, dchi=gchi)


def _exact_bonded(case, seed):
    s = _built(case, seed)
    x = torch.as_tensor(s["positions"], device="cuda").double().requires_grad_(True)
    box = torch.as_tensor(s["config"].box(), device="cuda")
    topo = _topo64(s["topology"])
    e, vir = _bond64(x, box, topo)
    force = lambda e: -torch.autograd.grad(e, x)[0]  # noqa: E731
    out = dict(e_bond=float(e), pr_bond=vir, f_bond=force(e))
    if len(topo[4]):
        e, vir = _angle64(x, box, topo)
        out.update(e_angle=float(e), pr_angle=vir, f_angle=force(e))
    if len(topo[9]):
        e = _dihedral64(x, box, topo)
        out.update(e_dihedral=float(e), f_dihedral=force(e), dipoles=None, transfer=None)
    return out


def _exact_gpe(case, seed):
    s = _built(case, seed)
    cfg = _gpe_config(s["config"])
    T = cfg.n_types
    m = _Mesh64(cfg.mesh(), cfg.box(), cfg.sigma)
    r = torch.as_tensor(s["positions"], device="cuda").double()
    t = torch.as_tensor(s["types"], device="cuda").long()
    q = torch.as_tensor(s["charges"], device="cuda").double()
    cic = m.cic(r)
    phi = m.c2r(m.r2c(m.paint(cic, t, torch.ones_like(q) / m.dV, T)) * m.H)
    rho = m.c2r(m.r2c(m.paint(cic, torch.zeros_like(t), q / m.dV, 1)) * m.H)[0]
    et = torch.tensor(cfg.dielectric_type, device="cuda", dtype=torch.float64)
    tot = phi.sum(0)
    eps = (et[:, None, None, None] * phi).sum(0) / tot
    q0 = rho / eps
    eta = m.c2r(1j * torch.stack([g * m.r2c(eps) for g in m.g])) / eps
    pol, delta, it = torch.zeros_like(rho), 1.0, 0
    while it < 100 and delta > cfg.conv_crit:
        E = m.gradient(m.r2c(q0 + pol) / m.kn)
        new = cfg.pol_mixing * -(eta * E).sum(0) + (1.0 - cfg.pol_mixing) * pol
        delta, pol, it = float((new - pol).abs().max()), new, it + 1
    e0 = COULOMB * 4.0 * math.pi
    psik = m.r2c(e0 * (q0 + pol)) / m.kn
    psi, E = m.c2r(psik), m.gradient(psik)
    dot = (E * E).sum(0)
    qt = torch.tensor(cfg.type_charges, device="cuda", dtype=torch.float64)
    vbar = [qt[k] * psi - 0.5 / e0 * (et[k] - eps) * dot / tot for k in range(T)]
    mesh = m.gradient(m.r2c(torch.stack(vbar)) * m.H)
    return dict(vbar=vbar, eps=eps, dot=dot, psi=psi, elec_field=list(E),
                f_elec=m.readout(cic, mesh, t))


def _exact_reverse(case, seed):
    s = _built(case, seed)
    cfg = s["config"]
    T, mass, dt, inner = cfg.n_types, float(cfg.mass), cfg.time_step, cfg.respa_inner
    m = _Mesh64(cfg.mesh(), cfg.box(), cfg.sigma)
    types = torch.as_tensor(s["types"], device="cuda")
    topo = _topo64(s["topology"])
    x0 = torch.as_tensor(s["positions"], device="cuda").double().requires_grad_(True)
    v0 = torch.as_tensor(s["velocities"], device="cuda").double().requires_grad_(True)
    chi = torch.tensor(_chi_matrix(cfg), device="cuda", requires_grad=True)
    rho0 = cfg.n_particles / m.V
    inc = 1.0 / (cfg.kappa * rho0)
    Q = inc + 0.5 * (chi + chi.T) * (1 - torch.eye(T, device="cuda").double()) / rho0
    t, box = types.long(), m.box

    def slow(x):
        cic = m.cic(x)
        spec = m.r2c(m.paint(cic, t, torch.ones_like(x[:, 0]) / m.dV, T)) * m.H
        v = torch.einsum("tj,jxyz->txyz", Q.to(spec.dtype), spec)
        return m.readout(cic, m.gradient(v * m.H), t)

    x, v = x0, v0
    ff, fb = slow(x), _bonded64(x, box, topo, True)[0]
    total = 0.0
    for _ in range(case["steps"]):
        v = v + 0.5 * inner * dt / mass * ff
        for _ in range(inner):
            v = v + 0.5 * dt / mass * fb
            x = torch.remainder(x + dt * v, box)
            fb = _bonded64(x, box, topo, True)[0]
            v = v + 0.5 * dt / mass * fb
        ff = slow(x)
        v = v + 0.5 * inner * dt / mass * ff
        z = x[:, 2] * (N_BINS / box[2]) - 0.5
        i0 = torch.floor(z).detach()
        f = z - i0
        i0 = i0.long() % N_BINS
        flat = torch.zeros(T * N_BINS, dtype=torch.float64, device="cuda")
        flat = flat.index_add(0, t * N_BINS + i0, 1.0 - f)
        flat = flat.index_add(0, t * N_BINS + (i0 + 1) % N_BINS, f)
        total = total + flat.reshape(T, N_BINS) / (m.V / N_BINS)
    prof = total / case["steps"]
    loss = ((prof - _target(case, cfg, seed).float().double()) ** 2).mean()
    gx, gv, gchi = torch.autograd.grad(loss, [x0, v0, chi])
    return dict(loss=loss.detach(), profile=prof.detach(), dx=gx, dv=gv, dchi=gchi)

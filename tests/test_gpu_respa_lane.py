"""The fused inner loop of small molecule groups (one bead, one bond and one
angle per lane) at the edges of what it takes: groups of exactly 32 beads,
molecules of 33, beads with 12 and 13 incidence entries, a single bond.

Forces against the real(8) restatement of the Fortran kernels (FP32 positions
and parameters; FP32 term arithmetic, 1e-5 relative RMS as for every bonded
kernel), and one outer step bit for bit against the general kernel (groups of
up to 64 beads), whose expressions it repeats in the same order.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import bonded as ob  # noqa: E402


def _system(shape, size, n_mol, seed=3):
    """n_mol chains of `size` beads, or stars of one bead and `size` arms,
    plus some free beads: (positions, velocities, types, packed, box)."""
    rng = np.random.default_rng(seed)
    box = np.array([6.0, 6.0, 6.0])
    per = size if shape == "chain" else size + 1
    if shape == "chain":
        bonds = [(i, i + 1) for i in range(per - 1)]
        angles = [(i, i + 1, i + 2) for i in range(per - 2)]
    else:
        bonds = [(0, 1 + i) for i in range(size)]
        angles = []
    pos = []
    for _ in range(n_mol):
        d = rng.normal(size=(per, 3))
        d *= 0.47 / np.linalg.norm(d, axis=1, keepdims=True)
        start = rng.uniform(0, 6, 3)
        pos.append(start + (np.cumsum(d, axis=0) if shape == "chain" else
                            np.concatenate([np.zeros((1, 3)), d[1:]])))
    free = rng.uniform(0, 6, (37, 3))
    r = np.mod(np.concatenate(pos + [free]) + rng.normal(0, 0.03, (per * n_mol + 37, 3)), box)
    off = per * np.arange(n_mol)
    b = (np.array(bonds)[None] + off[:, None, None]).reshape(-1, 2)
    a = (np.array(angles, dtype=int).reshape(-1, 3)[None] + off[:, None, None]).reshape(-1, 3)
    e = np.empty
    packed = (b[:, 0], b[:, 1], rng.uniform(0.4, 0.5, len(b)), np.full(len(b), 1250.0),
              a[:, 0], a[:, 1], a[:, 2], np.full(len(a), 2.0), np.full(len(a), 25.0),
              e(0, int), e(0, int), e(0, int), e(0, int), e((0, 6, 5)), e(0, int), e(0, int))
    v = rng.normal(0, 0.19, r.shape).astype(np.float32)
    types = (np.arange(len(r)) % 2).astype(np.int32)
    return np.mod(r.astype(np.float32), box.astype(np.float32)), v, types, packed, box


def _md(sys_, cap):
    from hymd_gb300.config import Config
    from hymd_gb300.hamiltonian import get_hamiltonian
    from hymd_gb300.md import RespaMD
    r, v, types, packed, box = sys_
    cfg = Config(n_steps=1, time_step=0.02, mesh_size=[16, 16, 16], sigma=0.5, kappa=0.05,
                 box_size=box, n_particles=len(r), n_types=2, mass=72.0, respa_inner=5,
                 hamiltonian="DefaultNoChi", m=[1.0, 1.0])
    md = RespaMD(r, v, types, cfg, get_hamiltonian(cfg), topology=packed, max_block_beads=cap)
    md.TUNE_SPECTRAL_TILE = False
    return md


@pytest.mark.parametrize("shape,size,n_mol", [
    ("chain", 2, 50), ("chain", 10, 7), ("chain", 16, 9), ("chain", 31, 5), ("chain", 32, 5),
    ("chain", 33, 4), ("star", 12, 6), ("star", 13, 6)])
def test_small_groups(shape, size, n_mol):
    sys_ = _system(shape, size, n_mol)
    r, _, _, packed, box = sys_
    small, large = _md(sys_, 32), _md(sys_, 64)
    small.prime()
    large.prime()
    got = small.f_b.cpu().numpy().astype(np.float64)
    fb, fa = np.zeros(r.shape), np.zeros(r.shape)
    x = r.astype(np.float64)
    p32 = [np.asarray(p, np.float32).astype(np.float64) if i in (2, 3, 7, 8) else p
           for i, p in enumerate(packed)]
    ob.compute_bond_forces(fb, x, box, *p32[0:4], precision="double")
    if len(packed[4]):
        ob.compute_angle_forces(fa, x, box, *p32[4:9], precision="double")
    ref = fb + fa
    err = np.sqrt(np.mean((got - ref) ** 2)) / np.sqrt(np.mean(ref ** 2))
    assert err < 1e-5, err
    assert torch.equal(small.f_b, large.f_b)
    for md in (small, large):
        md.step()
        md.check_errors()
    for name in ("r", "v", "f_b", "f_field"):
        assert torch.equal(getattr(small, name), getattr(large, name)), name

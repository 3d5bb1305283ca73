"""The per-term bonded kernels over their launch shapes (four-body terms: small
blocks up to one full block per SM, full ones beyond; all: several terms a
thread once the grid is full) against the FP64 C restatement.  Zigzag segments
away from the walls: a difference of two neighbouring positions is exact, a
bond's stretch of 0.05 carries 3e-8 / 0.05 = 6e-7 of rounding and the cosine
series and angles the same order, so forces agree to 1e-5 rel-RMS and energies
(sums of like-signed terms) to 1e-6."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import bonded as ob  # noqa: E402


def rel_rms(a, b):
    return float(np.sqrt(np.mean((np.asarray(a, np.float64) - b) ** 2) / np.mean(b ** 2)))


@pytest.mark.parametrize("n", [1, 63, 64, 65, 4097, 152 * 256, 152 * 256 + 1, 1024 * 256 + 65])
def test_terms_at_block_edges(n):
    from hymd_gb300 import force as gfo
    rng = np.random.default_rng(n)
    box = np.array([20.0, 21.0, 22.0])
    zig = np.array([[0, 0, 0], [0.45, 0.2, 0], [0.9, -0.1, 0.1], [1.3, 0.2, 0.4]])
    r = (rng.uniform(2.0, 17.0, (n, 1, 3)) + zig + rng.normal(0, 0.05, (n, 4, 3)))
    r = r.reshape(-1, 3).astype(np.float32)
    i = 4 * np.arange(n, dtype=np.int32)
    R, r64 = torch.as_tensor(r, device="cuda"), r.astype(np.float64)
    one = np.ones(n, np.float32)
    coeff = np.zeros((n, 6, 5), np.float32)
    coeff[:, 0], coeff[:, 1] = rng.uniform(1, 5, (n, 5)), rng.uniform(-3, 3, (n, 5))
    zero = np.zeros(n, np.int32)

    f, f64 = torch.zeros_like(R), np.zeros_like(r64)
    e, pr = gfo.compute_bond_forces(f, R, box, i, i + 1, 0.4 * one, 1250.0 * one)
    e64, pr64 = ob.compute_bond_forces(f64, r64, box, i, i + 1, 0.4 * one, 1250.0 * one,
                                       precision="double")
    assert rel_rms(f.cpu().numpy(), f64) < 1e-5
    assert e == pytest.approx(e64, rel=1e-6)
    assert np.allclose(pr, pr64, rtol=1e-5, atol=1e-5 * np.abs(pr64).max())

    f64 = np.zeros_like(r64)
    e, pr = gfo.compute_angle_forces(f, R, box, i, i + 1, i + 2, 1.5 * one, 100.0 * one)
    e64, _ = ob.compute_angle_forces(f64, r64, box, i, i + 1, i + 2, 1.5 * one, 100.0 * one,
                                     precision="double")
    assert rel_rms(f.cpu().numpy(), f64) < 1e-5
    assert e == pytest.approx(e64, rel=1e-6)

    f64 = np.zeros_like(r64)
    dip, tm = torch.zeros((n, 4, 3), device="cuda"), torch.zeros((n, 6, 3, 3), device="cuda")
    e = gfo.compute_dihedral_forces(f, R, dip, tm, box, i, i + 1, i + 2, i + 3, coeff, zero, zero,
                                    0)
    e64 = ob.compute_dihedral_forces(f64, r64, np.zeros((n, 4, 3)), np.zeros((n, 6, 3, 3)), box, i,
                                     i + 1, i + 2, i + 3, coeff, zero, zero, 0,
                                     precision="double")
    assert rel_rms(f.cpu().numpy(), f64) < 1e-5
    assert e == pytest.approx(e64, rel=1e-6)

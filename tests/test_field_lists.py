"""The lists of grids that the drop-in calls take are views of one stack, as many as the
call needs: a short or long list is refused (its stack would be filled beyond the grids
that were passed).  No GPU: host tensors in the place of device ones."""
import pytest

torch = pytest.importorskip("torch")


@pytest.fixture
def stack(monkeypatch):
    from hymd_gb300 import _lib, field
    monkeypatch.setattr(_lib, "require_cuda", lambda t, *a: t)
    return lambda lst, lead: field._stack_base(lst, lead, torch.float32, "phi")


def test_number_of_grids(stack):
    base = torch.arange(2 * 3 * 8.0).reshape(2, 3, 2, 2, 2)
    nested = [[base[t, d] for d in range(3)] for t in range(2)]
    got = stack(nested, (2, 3))
    assert got.shape == base.shape and got.data_ptr() == base.data_ptr()
    assert torch.equal(got, base)
    assert torch.equal(stack([tuple(x) for x in nested], (2, 3)), base)
    assert torch.equal(stack([nested], (2, 3)), base)
    flat = [base[t, d] for t in range(2) for d in range(3)]
    assert torch.equal(stack(flat, (6,)), base.reshape(6, 2, 2, 2))
    for lst, lead in ((flat[:1], (2,)), (flat[:5], (2, 3)), (flat, (5,)), (nested[:1], (2, 3)),
                      (nested, (2,)), ([nested[0][:2]], (3,)), ([], (1,))):
        with pytest.raises((ValueError, IndexError)):
            stack(lst, lead)
    with pytest.raises(ValueError):
        stack([flat[1], flat[0]], (2,))

"""Deferred rRESPA sums (hpf_respa_plan_defer) whose step stops between the inner
loop and the field step: the plan destroyed first, the rest of the step recorded in a
graph, another inner loop on the same plan, a field step that takes no deposits.
Every result has the bits of the same calls with the sums in stream order."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _md():
    from hymd_gb300 import systems
    from hymd_gb300.hamiltonian import get_hamiltonian
    from hymd_gb300.md import RespaMD
    s = systems.homopolymer_melt(seed=4, n_chains=150, length=10, box=5.6, mesh=24)
    md = RespaMD(s["positions"], s["velocities"], s["types"], s["config"],
                 get_hamiltonian(s["config"]), topology=s["topology"], max_block_beads=24)
    md.TUNE_SPECTRAL_TILE = False
    md.couple(thermostat=True, seed=3, n_steps=30)
    md.prime()
    md.step()
    assert md._defer_sums
    return md


def _same(a, b):
    torch.cuda.synchronize()
    a.check_errors()
    for name in ("r", "v", "f_b", "f_field", "bonded_out", "state"):
        assert torch.equal(getattr(a, name), getattr(b, name)), name


def _inner(md, defer):
    from hymd_gb300 import _lib
    md._inner_fused(_lib.stream_ptr(), defer=defer)


def _rest(md):
    from hymd_gb300 import _lib
    md._outer_rest(_lib.stream_ptr())


def test_plan_destroyed_before_the_field_step():
    from hymd_gb300 import _lib
    out = []
    for defer in (True, False):
        md = _md()
        _inner(md, defer)
        plan, md.plan = md.plan, md._make_plan(md._packed, md.block_beads)
        _lib.lib().hpf_respa_plan_destroy(plan)
        _rest(md)
        md.step()
        out.append(md)
    _same(*out)


def test_rest_of_the_step_in_a_graph():
    out = []
    for defer in (True, False):
        md = _md()
        _inner(md, defer)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            _rest(md)
        g.replay()
        md.step()
        out.append(md)
    _same(*out)


def test_two_inner_loops():
    out = []
    for defer in (True, False):
        md = _md()
        _inner(md, defer)
        _inner(md, defer)
        _rest(md)
        out.append(md)
    _same(*out)


def test_context_destroyed_first():
    """The plan outlives its mesh context, and the other way round."""
    from hymd_gb300 import _lib
    for first in ("pm", "plan"):
        md = _md()
        _inner(md, True)
        torch.cuda.synchronize()
        if first == "pm":
            _lib.lib().hpf_ctx_destroy(md.pm._h)
            md.pm._h = None
            _lib.lib().hpf_respa_plan_destroy(md.plan)
            md.plan = None
        else:
            _lib.lib().hpf_respa_plan_destroy(md.plan)
            md.plan = None
            _lib.lib().hpf_ctx_destroy(md.pm._h)
            md.pm._h = None

"""Fields of the fused form read one after another."""
import pytest
import torch

from tests.gpu_util import init_with, lbm_config, require_cuda, run, smooth_f0

pytestmark = pytest.mark.gpu
W, P = 1200, 11000


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    require_cuda()


def _stepped(storage="fp32"):
    from funlbm_b200.lbm import LBMD3

    lbm = LBMD3(config=lbm_config(19, (12, 10, 14), 0.08, [W, W, P, P, W, W],
                                  body_force=(1e-5, 0, 0), storage=storage))
    init_with(lbm, smooth_f0(19, (13, 11, 15), 0.03, 5))
    run(lbm, 3)
    return lbm


@pytest.mark.parametrize("storage", ["fp32", "fp16s"])
def test_f_brings_u_and_rho(storage):
    """f, then u and rho: one read of the populations; the same values as read
    in another order."""
    a, b = _stepped(storage), _stepped(storage)
    calls = []
    plain = a.flow.lattice.observe
    a.flow.lattice.observe = lambda *args, **kw: (calls.append(1), plain(*args, **kw))
    first = [a.flow.f, a.flow.u, a.flow.rou]
    assert len(calls) == 1
    rou, u, f = b.flow.rou, b.flow.u, b.flow.f
    for x, y in zip(first, (f, u, rou)):
        assert torch.equal(x, y)


@pytest.mark.parametrize("write", [
    lambda rou: rou.sub_(1.0),
    lambda rou: rou[3:, ..., 0].zero_(),
    lambda rou: rou.view(-1)[::2].fill_(5.0),
])
def test_p_of_a_rho_that_was_written_to(write):
    a, b = _stepped(), _stepped()
    want = a.flow.p.clone()
    rou = b.flow.rou
    kept = rou.clone()
    write(rou)
    mine = rou.clone()
    assert torch.equal(b.flow.p, want)
    assert torch.equal(want, kept / 3.0)
    assert torch.equal(b.flow.rou, mine)            # what the caller wrote stays
    run(b, 1)
    run(a, 1)
    assert torch.equal(b.flow.rou, a.flow.rou) and torch.equal(b.flow.p, a.flow.p)


def test_p_in_inference_mode():
    with torch.inference_mode():
        a, b = _stepped(), _stepped()
        want = a.flow.p.clone()
        b.flow.rou.zero_()
        assert torch.equal(b.flow.p, want)


@pytest.mark.parametrize("when", ["before", "between"])
def test_force_field_written_through_a_kept_reference(when):
    """Reference call sequence: FOL taken before or between steps and written to
    in place is cleared within the next step, as when no pass is skipped."""
    from funlbm_b200.lbm import LBMD3

    def stepped(skip):
        lbm = LBMD3(config=lbm_config(19, (9, 6, 7), 0.1, [1400, 1400, W, W, W, W]))
        init_with(lbm, smooth_f0(19, (10, 7, 8), 0.02, 2))
        if not skip:
            lbm._no_force = lambda: False
        if when == "between":
            run(lbm, 2)
        fol = lbm.flow.FOL
        run(lbm, 3)
        states = []
        for _ in range(3):
            fol.fill_(1e-4)
            run(lbm, 1)
            states += [lbm.flow.f.clone(), lbm.flow.u.clone(), lbm.flow.rou.clone(), fol.clone()]
        return states

    for a, b in zip(stepped(True), stepped(False)):
        assert torch.equal(a, b)


def test_forcing_is_skipped_until_the_force_field_is_handed_out(tmp_path):
    from funlbm_b200.lbm import LBMD3, _NpzGroup

    lbm = LBMD3(config=lbm_config(19, (9, 6, 7), 0.1, [1400, 1400, W, W, W, W]))
    lbm.init()
    run(lbm, 2)
    assert lbm._no_force()
    store = _NpzGroup()
    lbm.dump_checkpoint(store)                      # (reads FOL, hands nothing out)
    run(lbm, 1)
    assert lbm._no_force()
    other = LBMD3(config=lbm_config(19, (9, 6, 7), 0.1, [1400, 1400, W, W, W, W]))
    other.init()
    other.load_checkpoint(group=store)
    run(other, 1)
    assert other._no_force()
    lbm.flow.FOL
    run(lbm, 2)
    assert not lbm._no_force()


@pytest.mark.parametrize("q", [13, 19, 27])
@pytest.mark.parametrize("faces", [[1400, 1400, W, W, W, W], [1400, W, P, P, W, W],
                                   [P, P, W, W, P, P], [W, W, W, W, W, 1201]])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf"), "empty"])
def test_steps_without_force_keep_what_is_not_finite(q, faces, bad):
    """Populations that are not finite, and nodes of density zero, spread in the
    steps that skip the forcing as they do through it."""
    from funlbm_b200.lbm import LBMD3

    shape = (10, 7, 8)

    def stepped(skip):
        lbm = LBMD3(config=lbm_config(q, (9, 6, 7), 0.1, faces, uw=[(0.0, 0.01, 0.0)] * 6,
                                      fused=False))
        f0 = torch.tensor(smooth_f0(q, shape, 0.02, 2))
        for k, at in enumerate([(4, 3, 4), (8, 3, 3), (1, 2, 2), (0, 3, 5)]):
            if bad == "empty":
                f0[at] = 0.0
            else:
                f0[at][3 + k] = bad
        init_with(lbm, f0.numpy())
        if not skip:
            lbm._no_force = lambda: False
        states = []
        for _ in range(3):
            run(lbm, 1)
            states += [getattr(lbm.flow, k).clone() for k in ("f", "u", "rou", "p")]
        return states

    for k, (a, b) in enumerate(zip(stepped(True), stepped(False))):
        assert torch.equal(torch.isnan(a), torch.isnan(b)), k
        assert torch.equal(torch.nan_to_num(a, nan=0.0), torch.nan_to_num(b, nan=0.0)), k


def _counted(calls, name, method):
    def call(self, *args, **kw):
        calls.append(name)
        return method(self, *args, **kw)
    return call


@pytest.mark.parametrize("name", ["cul_equ", "f_stream", "update_u_rou", "cul_equ2"])
def test_flow_methods_replaced_on_the_class_are_called(monkeypatch, name):
    from funlbm_b200.flow import FlowD3
    from funlbm_b200.lbm import LBMD3

    lbm = LBMD3(config=lbm_config(19, (9, 6, 7), 0.1, [1400, 1400, W, W, W, W]))
    lbm.init()
    run(lbm, 1)
    calls = []
    monkeypatch.setattr(FlowD3, name, _counted(calls, name, getattr(FlowD3, name)))
    run(lbm, 3)
    assert len(calls) == (6 if name == "update_u_rou" else 3)


@pytest.mark.parametrize("name", ["flow_to_lagrange", "particle_to_wall", "lagrange_to_flow"])
def test_coupling_methods_replaced_on_the_class_are_called(monkeypatch, name):
    from funlbm_b200.lbm import LBMD3

    lbm = LBMD3(config=lbm_config(19, (9, 6, 7), 0.1, [1400, 1400, W, W, W, W]))
    lbm.init()
    run(lbm, 1)
    calls = []
    monkeypatch.setattr(LBMD3, name, _counted(calls, name, getattr(LBMD3, name)))
    run(lbm, 3)
    assert len(calls) == 3


@pytest.mark.parametrize("how", ["class", "subclass", "instance"])
@pytest.mark.parametrize("owner,name", [("lbm", "fused_prepare"), ("lbm", "fused_finish"),
                                        ("flow", "enter_fused"), ("flow", "fused_step"),
                                        ("lattice", "step")])
def test_step_methods_replaced_in_particle_runs_are_called(monkeypatch, owner, name, how):
    """A particle step goes through the methods of the fused step when one of
    them is replaced, with the same results."""
    from funlbm_b200.lbm import LBMD3

    def make():
        lbm = LBMD3(config=lbm_config(19, (24, 18, 20), 0.08, [W, W, P, P, W, W], gl=1e-3,
                                      particles=[{"type": "sphere", "r": 3, "rou": 1.4,
                                                  "coord": {"center": [12, 9, 10]}}]))
        lbm.init()
        run(lbm, 2)
        return lbm

    a, b = make(), make()
    run(a, 3)
    obj = {"lbm": b, "flow": b.flow, "lattice": b.flow.lattice}[owner]
    calls = []
    cls = type(obj)
    counted = _counted(calls, name, getattr(cls, name))
    if how == "class":
        monkeypatch.setattr(cls, name, counted)
    elif how == "subclass":
        obj.__class__ = type("Own", (cls,), {name: counted})
    else:
        monkeypatch.setattr(obj, name, lambda *args, **kw: counted(obj, *args, **kw))
    run(b, 3)
    assert len(calls) == 3
    assert torch.equal(a.flow.u, b.flow.u)
    assert torch.equal(a.particle_swarm.lx, b.particle_swarm.lx)


@pytest.mark.parametrize("how,made", [("run_step", True), ("run_steps", True), ("packed", False),
                                      ("accumulate", False)])
def test_boxes_are_allocated_for_the_steps_that_use_them(how, made):
    """The scratch of the node moments belongs to the combined particle step;
    steps packed with other lattices and the accumulating mode do without."""
    from funlbm_b200.lbm import LBMD3

    lbm = LBMD3(config=lbm_config(19, (24, 18, 20), 0.08, [W, W, P, P, W, W], gl=1e-3,
                                  ibm_mode="accumulate" if how == "accumulate" else "reference",
                                  particles=[{"type": "sphere", "r": 4, "rou": 1.4,
                                              "coord": {"center": [12, 9, 10]}}]))
    lbm._BOX_MARKERS = 1
    lbm.init()
    if how == "packed":
        for _ in range(3):
            plan = lbm.fused_prepare()
            lbm.flow.fused_step(plan["force"], plan["new_field"], plan["g_new"], keep=plan["keep"])
            lbm.fused_finish(plan)
            lbm.step += 1
    elif how == "run_steps":
        lbm.run_steps(40)
    else:
        run(lbm, 3)
    assert (lbm._boxes is not None) == made
    assert float(lbm.flow.u.abs().max()) > 0 and lbm.check_status() == 0


@pytest.mark.parametrize("storage", ["fp32", "bf16s", "fp64"])
@pytest.mark.parametrize("g", [(0, 0, 0), (1e-5, 0, 0), (0.1, -0.2, 0.3)])
def test_force_field_of_a_fused_run(storage, g):
    """FOL of a run with a uniform force alone: the force as float32 at every
    node, made without a copy from the host."""
    from funlbm_b200.lbm import LBMD3

    lbm = LBMD3(config=lbm_config(19, (6, 5, 7), 0.3, [P] * 6, body_force=g, storage=storage))
    lbm.init()
    run(lbm, 2)
    torch.cuda.synchronize()
    mode = torch.cuda.get_sync_debug_mode()
    torch.cuda.set_sync_debug_mode("error")
    try:
        fol = lbm.flow.FOL
    finally:
        torch.cuda.set_sync_debug_mode(mode)
    assert fol.dtype == lbm.flow.lattice.real_dtype and fol.shape == (7, 6, 8, 3)
    assert fol.is_contiguous()
    assert torch.equal(fol[..., :].cpu().float(), torch.tensor(g, dtype=torch.float32).expand(7, 6, 8, 3))

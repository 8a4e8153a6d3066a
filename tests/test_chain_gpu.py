"""Observations queued between chained steps: every field equals the one of a
run that waits for the device after each call."""
import pytest
import torch

from tests.gpu_util import init_with, lbm_config, require_cuda, smooth_f0

pytestmark = pytest.mark.gpu
W, P = 1200, 11000


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    require_cuda()


@pytest.mark.parametrize("storage", ["fp32", "fp16s"])
@pytest.mark.parametrize("shape,steps", [
    ((24, 20, 31), 32),          # all blocks of a step resident at once
    ((256, 256, 256), 6),
])
def test_observed_steps_in_a_queue(storage, shape, steps):
    """Lattice.step with observation buffers, many in a row."""
    from funlbm_b200.lattice import Lattice, make_force, tau_float32

    f0 = torch.tensor(smooth_f0(19, shape, 0.05, 3)).cuda().permute(3, 0, 1, 2).reshape(19, -1)
    force = make_force((1e-5, 0, 0), (1e-5, 0, 0))

    def run(wait):
        lat = Lattice(19, shape, [P, P, P, P, W, W], tau_float32(0.05), storage=storage)
        lat.init(f0.contiguous())
        out = [(torch.zeros(lat.n, device="cuda"), torch.zeros(lat.n, 3, device="cuda"))
               for _ in range(steps)]
        torch.cuda.synchronize()
        from funlbm_b200._lib import LbmObserve, ptr

        for rho, u in out:
            lat.step(force, obs=LbmObserve(None, ptr(rho), ptr(u)))
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        assert lat.read_status() == 0
        return out

    for k, (a, b) in enumerate(zip(run(True), run(False))):
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1]), k


@pytest.mark.parametrize("particles", [False, True])
def test_fields_read_between_queued_steps(particles):
    """u and f read after every run_step, without a host synchronisation."""
    from funlbm_b200.lbm import LBMD3

    parts = [{"type": "sphere", "r": 3, "rou": 1.4, "coord": {"center": [12, 9, 10]}}]

    def run(wait):
        lbm = LBMD3(config=lbm_config(19, (24, 18, 20), 0.08, [W, W, P, P, W, W], gl=1e-3,
                                      body_force=(1e-6, 0, 0), particles=parts if particles else ()))
        init_with(lbm, smooth_f0(19, (25, 19, 21), 0.03, 5))
        lat_out = []
        for _ in range(24):
            lbm.run_step(step=lbm.step)
            lbm.step += 1
            lat_out.append((lbm.flow.u.clone(), lbm.flow.f.clone()))
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return lat_out

    for k, (a, b) in enumerate(zip(run(True), run(False))):
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1]), k


def test_steps_around_a_read_stay_in_order():
    """step, observe into a buffer, step, ... with nothing else in the stream."""
    from funlbm_b200.lattice import Lattice, tau_float32

    shape = (40, 36, 33)
    f0 = torch.tensor(smooth_f0(19, shape, 0.05, 7)).cuda().permute(3, 0, 1, 2).reshape(19, -1)

    def run(wait):
        lat = Lattice(19, shape, [P] * 6, tau_float32(0.05))
        lat.init(f0.contiguous())
        rho, u = torch.zeros(lat.n, device="cuda"), torch.zeros(lat.n, 3, device="cuda")
        for _ in range(200):
            lat.step()
            lat.observe(None, rho=rho, u=u)
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return lat.buf[lat.cur].view(19, -1, lat.pz)[:, :, :shape[2]].clone(), rho, u

    for a, b in zip(run(True), run(False)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("storage", ["fp32", "fp16s", "bf16s", "fp64"])
@pytest.mark.parametrize("nz,pitch,nodes", [
    (33, None, 0), (33, False, 0), (33, False, 1), (32, None, 0), (32, None, -1), (32, True, 2),
])
def test_observed_step_is_one_launch(storage, nz, pitch, nodes):
    """A step with observation buffers reads the populations once and gives
    what the step and the observation give apart."""
    runtime = pytest.importorskip("cuda.bindings.runtime")
    from funlbm_b200._lib import LbmObserve, ptr
    from funlbm_b200.lattice import Lattice, make_force, tau_float32

    if storage == "fp64" and nodes == -1:
        pytest.skip("row staging is not built for FP64")
    S = 1201
    shape = (9, 7, nz)
    lat = Lattice(19, shape, [W, S, P, P, W, S], tau_float32(0.05), storage=storage, pitch=pitch,
                  face_uw=[(0.01, -0.02, 0.015)] * 6)
    lat.set_launch_shape(nodes, 128)
    dt = lat.real_dtype
    lat.init(torch.tensor(smooth_f0(19, shape, 0.05, 2)).cuda().permute(3, 0, 1, 2)
             .reshape(19, -1).to(dt).contiguous())
    force = make_force((1e-5, 0, 0), (0, 2e-5, 0))
    lat.step(force)

    def fields():
        return [torch.zeros(s, dtype=dt, device="cuda") for s in ((19, lat.n), (lat.n,), (lat.n, 3))]

    def stored(b):
        return b.view(19, -1, lat.pz)[:, :, :nz].clone()

    lat.step(force)                                   # apart
    apart = fields()
    lat.observe(force, *apart)
    after, rho_after = stored(lat.buf[lat.cur]), lat.face_rho[lat.cur].clone()
    lat.cur ^= 1
    lat.buf[lat.cur ^ 1].zero_()
    lat.face_rho[lat.cur ^ 1].zero_()
    both = fields()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        g.capture_begin()
        lat.step(force, obs=LbmObserve(*(ptr(t) for t in both)))
        g.capture_end()
    err, _, count = runtime.cudaGraphGetNodes(runtime.cudaGraph_t(init_value=g.raw_cuda_graph()), 0)[:3]
    assert int(err) == 0 and count == 1
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    for a, b in zip(apart, both):
        assert torch.equal(a, b)
    assert torch.equal(after, stored(lat.buf[lat.cur]))
    assert torch.equal(rho_after, lat.face_rho[lat.cur])
    assert lat.read_status() == 0

"""Launch forms against each other, bit for bit: node pairs in packed
arithmetic against one node per thread, the combined library calls against the
calls they stand for, fields observed one at a time against all at once."""
import ctypes

import numpy as np
import pytest
import torch

from tests.gpu_util import init_with, lbm_config, require_cuda, run, smooth_f0

pytestmark = pytest.mark.gpu
W, P, S = 1200, 11000, 1201


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    require_cuda()


def _forced_run(q, storage, shape, faces, pitch, nodes, seed):
    """Five steps under a body force and random force fields in random 32-node
    chunks; f, rho and u of the last one."""
    from funlbm_b200.lattice import Lattice, make_force, tau_float32

    g = torch.Generator().manual_seed(seed)
    lat = Lattice(q, shape, faces, tau_float32(0.06), storage=storage, pitch=pitch,
                  face_uw=[(0.01 * i, -0.02, 0.015) for i in range(6)])
    lat.set_launch_shape(nodes, 128)
    lat.init(torch.tensor(smooth_f0(q, shape, 0.05, seed)).cuda().permute(3, 0, 1, 2).contiguous()
             .view(q, -1))
    fields, flags = [], []
    for _ in range(2):
        fl = (torch.rand((lat.n + 31) // 32, generator=g) < 0.4).to(torch.uint8)
        f = 1e-4 * torch.randn(lat.n, 3, generator=g)
        f *= (torch.rand(lat.n, 1, generator=g) < 0.5) * fl.repeat_interleave(32)[:lat.n, None]
        fields.append(f.cuda().reshape(-1))
        flags.append(fl.cuda())
    for k in range(5):
        old, new = k % 2, 1 - k % 2
        force = make_force((0, 0, 0), (0, 0, 0) if k < 3 else (1e-5, 0, -2e-5), fields[old],
                           fields[new], flags[old], flags[new])
        lat.step(force)
    out = [torch.empty((q, lat.n), device="cuda"), torch.empty(lat.n, device="cuda"),
           torch.empty((lat.n, 3), device="cuda")]
    lat.observe(force, *out)
    for k in range(3):       # each of them alone
        one = [None, None, None]
        one[k] = torch.empty_like(out[k])
        lat.observe(force, *one)
        assert torch.equal(one[k], out[k]), k
    assert lat.read_status() == 0
    return [t.cpu().numpy() for t in out]


@pytest.mark.parametrize("storage", ["fp32", "fp16s", "bf16s"])
@pytest.mark.parametrize("q", [13, 15, 19, 27])
@pytest.mark.parametrize("shape,faces", [
    ((6, 5, 33), [W, P, P, W, S, W]),      # rows padded by one, a partial last pair
    ((5, 9, 35), [S, W, W, S, P, P]),
    ((4, 7, 5), [P] * 6),                  # a row of three pairs
    ((5, 6, 32), [P, P, S, W, W, S]),      # even rows, no padding
])
def test_pairs_equal_single_nodes(q, storage, shape, faces):
    dense = _forced_run(q, storage, shape, faces, False, 1, 3)
    forms = [(None, 2), (True, 2)]
    if storage != "fp32" or shape[2] > 8:
        forms.append((True, 4))
    for pitch, nodes in forms:
        got = _forced_run(q, storage, shape, faces, pitch, nodes, 3)
        for a, b in zip(dense, got):
            assert np.array_equal(a, b), (pitch, nodes)


@pytest.mark.parametrize("q", [13, 19, 27])
@pytest.mark.parametrize("faces", [[1400, 1400, W, W, W, W], [1400, W, P, P, W, S], [W, P, S, W, P, P]])
def test_compute_flow_equals_its_calls(q, faces):
    from funlbm_b200.lbm import LBMD3

    def flow():
        lbm = LBMD3(config=lbm_config(q, (9, 6, 11), 0.1, faces,
                                      uw=[(0.01, 0.02, -0.01)] * 6, fused=False))
        init_with(lbm, smooth_f0(q, (10, 7, 12), 0.03, 5))
        lbm.flow.FOL = 1e-5 * torch.randn((10, 7, 12, 3), generator=torch.Generator().manual_seed(1))
        return lbm.flow

    a, b = flow(), flow()
    for _ in range(3):
        a.compute_flow()
        b.cul_equ()
        b.f_stream()
        b.update_u_rou()
        for k in ("f", "rou", "u", "p", "feq"):
            assert torch.equal(getattr(a, k), getattr(b, k)), k


def test_no_force_step_skips_nothing_that_counts():
    """Non-equilibrium channel: steps that skip the forcing pass against steps
    that run it on a FOL of zeros, and a replaced method is still called."""
    from funlbm_b200.lbm import LBMD3

    def make():
        lbm = LBMD3(config=lbm_config(19, (9, 6, 7), 0.1, [1400, 1400, W, W, W, W]))
        init_with(lbm, smooth_f0(19, (10, 7, 8), 0.02, 2))
        return lbm

    a, b, c = make(), make(), make()
    calls = []
    plain = b.lagrange_to_flow
    b.lagrange_to_flow = lambda *args: (calls.append(1), plain(*args))
    c.flow.FOL = 1e-4 * torch.ones((10, 7, 8, 3))       # dropped by the first step's spreading
    for lbm in (a, b, c):
        run(lbm, 4)
    assert len(calls) == 4
    for k in ("f", "rou", "u"):
        assert torch.equal(getattr(a.flow, k), getattr(b.flow, k)), k
    assert float(c.flow.FOL.abs().max()) == 0.0


@pytest.mark.parametrize("storage", ["fp32", "fp16s", "fp64"])
def test_coupled_step_equals_its_calls(storage):
    from funlbm_b200.lbm import LBMD3

    parts = [{"type": "sphere", "r": 3, "rou": 1.3, "coord": {"center": [12, 9, 9]}},
             {"type": "ellipsoid", "a": 4, "b": 2, "c": 2, "rou": 1.1,
              "coord": {"center": [18, 8, 10], "alpha": 0.3, "beta": 0.5, "gamma": 0.1}}]

    def make():
        lbm = LBMD3(config=lbm_config(19, (24, 18, 20), 0.08, [W, W, P, P, W, W], gl=1e-3,
                                      storage=storage, particles=parts, body_force=(0, 1e-6, 0)))
        lbm.init()
        return lbm

    a, b = make(), make()
    b._coupled_step = lambda: False
    for lbm in (a, b):
        run(lbm, 7)
    for k in ("f", "u", "rou", "FOL"):
        assert torch.equal(getattr(a.flow, k), getattr(b.flow, k)), k
    for k in ("lx", "lF", "cx", "cu", "cw", "angle", "extreme"):
        assert torch.equal(getattr(a.particle_swarm, k), getattr(b.particle_swarm, k)), k


@pytest.mark.parametrize("storage", ["fp32", "bf16s", "fp64"])
@pytest.mark.parametrize("cells", [None, 900, 60])
def test_box_moments_equal_slot_moments(storage, cells):
    """Interpolation from moments taken once per node: bodies of two sizes, one
    across a wall, boxes that do not fit (60: none does, 900: the small
    body's only)."""
    from funlbm_b200.lbm import LBMD3

    parts = [{"type": "sphere", "r": 4, "rou": 1.3, "coord": {"center": [12, 9, 9]}},
             {"type": "sphere", "r": 2, "rou": 1.3, "coord": {"center": [4, 12, 16]}},
             {"type": "ellipsoid", "a": 4, "b": 3, "c": 2, "rou": 0.9,
              "coord": {"center": [23, 16, 2], "alpha": 0.3, "beta": 0.5, "gamma": 0.1}}]

    def make(least):
        lbm = LBMD3(config=lbm_config(19, (25, 19, 20), 0.08, [W, W, P, P, W, S], gl=1e-3,
                                      uw=[(0.0, 0.01, 0.0)] * 6, storage=storage, particles=parts))
        lbm._BOX_MARKERS = least
        lbm.init()
        return lbm

    a, b = make(1), make(10 ** 9)
    for k in range(8):
        if k == 2 and cells is not None:
            a._boxes = (a._boxes[0], cells, 3)
        if k == 5:          # positions moved in place: the extremes are stale
            for lbm in (a, b):
                lbm.particle_swarm.lx[:40] += 5.0
        for lbm in (a, b):
            run(lbm, 1)
    assert a._boxes is not None and b._boxes is None
    for k in ("f", "u", "rou", "FOL"):
        assert torch.equal(getattr(a.flow, k), getattr(b.flow, k)), k
    for k in ("lx", "lF", "lu", "lrou", "cx", "cu", "cw"):
        assert torch.equal(getattr(a.particle_swarm, k), getattr(b.particle_swarm, k)), k


def test_coupled_step_refuses_what_it_needs():
    from funlbm_b200 import _lib
    from funlbm_b200.lattice import Lattice, make_force

    lat = Lattice(19, (8, 8, 8), [W] * 6, 0.7)
    pt = _lib.LbmParticles()
    pt.n_particles, pt.n_markers = 1, 1
    with pytest.raises(ValueError):
        _lib.call("lbm_coupled_step", ctypes.byref(lat.desc), lat.buf[0].data_ptr(),
                  lat.buf[1].data_ptr(), ctypes.byref(make_force()), None, None, ctypes.byref(pt),
                  1.0, 1.0, 0.0, 1.0, 1, None, None, 0, 0, None, None, lat.stream())


@pytest.mark.parametrize("storage", ["fp32", "bf16s"])
@pytest.mark.parametrize("shape", [(6, 5, 33), (5, 9, 3), (4, 6, 35), (7, 4, 129), (5, 6, 32)])
@pytest.mark.parametrize("pitch", [None, True])
@pytest.mark.parametrize("step", [False, True])
def test_observed_fields_at_odd_places(storage, shape, pitch, step):
    """Pairs of odd rows, and buffers that begin at odd places, against one node
    per thread; the floats around the buffers keep their values."""
    from funlbm_b200._lib import LbmObserve
    from funlbm_b200.lattice import Lattice, tau_float32

    q, n = 15, shape[0] * shape[1] * shape[2]
    f0 = torch.tensor(smooth_f0(q, shape, 0.05, 9)).cuda().permute(3, 0, 1, 2).reshape(q, -1)

    def fields(nodes, pitch, off):
        lat = Lattice(q, shape, [W, P, P, P, W, W], tau_float32(0.06), storage=storage, pitch=pitch)
        lat.init(f0.contiguous())
        lat.step()
        lat.set_launch_shape(nodes, 128)
        out = [torch.full((k * n + 8,), -7.0, device="cuda") for k in (q, 1, 3)]
        obs = LbmObserve(*(t.data_ptr() + 4 * (off + j) for j, t in enumerate(out)))
        if step:
            lat.step(obs=obs)
        else:
            lat.step()
            lat.cur ^= 1
            from funlbm_b200._lib import call, ctypes, ptr

            call("lbm_flow_step", ctypes.byref(lat.desc), ptr(lat.buf[lat.cur]), None, None, None,
                 None, ctypes.byref(obs), None, lat.stream())
        got = []
        for j, (t, k) in enumerate(zip(out, (q, 1, 3))):
            lo = off + j
            got.append(t[lo:lo + k * n].clone())
            assert bool((t[:lo] == -7).all()) and bool((t[lo + k * n:] == -7).all())
        return got

    want = fields(1, False, 0)
    for off in (0, 1, 2):
        for a, b in zip(want, fields(0, pitch, off)):
            assert torch.equal(a, b)


@pytest.mark.parametrize("storage", ["fp16s", "bf16s"])
@pytest.mark.parametrize("nz,pitch", [(33, 35), (32, 33), (4, 7)])
def test_two_nodes_on_rows_of_odd_pitch(storage, nz, pitch):
    """Two nodes per thread asked for on padded rows of odd pitch: the same bits
    as on dense rows."""
    shape, faces = (6, 5, nz), [W, P, P, W, S, W]
    dense = _forced_run(19, storage, shape, faces, False, 1, 3)
    for a, b in zip(dense, _forced_run(19, storage, shape, faces, pitch, 2, 3)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("storage", ["fp32", "fp16s", "bf16s", "fp64"])
@pytest.mark.parametrize("pitch", [None, 35, True])
def test_entering_padded_rows(storage, pitch):
    """lbm_flow_init and load_post_collision_fp32 on padded rows against dense
    rows and against torch; init writes the padding."""
    from funlbm_b200.lattice import FP16_SCALE, STORAGE_DTYPE, Lattice, weights_tensor

    shape = (6, 5, 33)
    f = torch.tensor(smooth_f0(19, shape, 0.05, 4)).cuda().permute(3, 0, 1, 2).reshape(19, -1)

    def rows(pitch, load):
        lat = Lattice(19, shape, [W, P, P, W, W, W], 0.7, storage=storage, pitch=pitch)
        for b in lat.buf:
            b.fill_(float("nan"))
        g = f.to(lat.real_dtype).contiguous()
        lat.load_post_collision_fp32(g) if load else lat.init(g)
        all_rows = lat.buf[lat.cur].view(19, -1, lat.pz)
        return all_rows[:, :, :33].clone(), all_rows[:, :, 33:].clone()

    for load in (False, True):
        a, b = rows(False, load), rows(pitch, load)
        assert torch.equal(a[0], b[0]) and not bool(b[0].isnan().any())
        if not load:
            assert not bool(b[1].isnan().any())
    d = f.view(19, 30, 33).double() if storage == "fp64" else f.view(19, 30, 33) - weights_tensor(
        19, f.device)[:, None, None]
    if storage == "fp16s":
        d = d * FP16_SCALE
    assert torch.equal(rows(pitch, True)[0], d.to(STORAGE_DTYPE[storage]))

"""ops.active_list and ops.update_list against the mask op and torch.nonzero, at
the edges of their 4096-cell blocks and 32-cell words, and through the solver
object against the op-by-op loop."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 4095, 4096, 4097, 8192, 300_001])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("share", [0.0, 0.02, 0.7, 1.0])
def test_lists_equal_nonzero(cuda, n, dtype, share):
    from hipims_b200 import ops

    rng = np.random.default_rng(n)
    h = torch.as_tensor(np.where(rng.uniform(size=n) < share, rng.uniform(0, 1, n), 0.0),
                        dtype=dtype, device=cuda)
    hs = torch.tensor(1.0e-6, dtype=dtype, device=cuda)
    h[rng.integers(0, n, max(n // 50, 1))] = hs          # exactly the dry depth: dry
    index = torch.as_tensor(np.concatenate([np.full(n, 10), rng.integers(-1, n, 4 * n)]),
                            dtype=torch.int32, device=cuda)
    for t in (0.0, 3.0):
        tt = torch.tensor([t], dtype=dtype, device=cuda)
        mask = torch.zeros(n, dtype=torch.bool, device=cuda)
        ops.flux_mask(mask, h, index, tt)
        want = mask.nonzero().flatten().to(torch.int32)
        got = ops.active_list(h, index, tt)
        assert got.dtype == torch.int32 and torch.equal(got, want)
    u = torch.where(torch.rand(n, device=cuda) < share, torch.randn(n, device=cuda), 0.0).to(dtype)
    x = torch.where(torch.rand(n, device=cuda) < 0.5, -h - 1.0, h)
    if n > 3:
        x[0], u[1], x[2], u[2] = float("nan"), float("nan"), -1.0, float("inf")
    want = ((u.abs() > 0) | (x >= 0)).nonzero().flatten().to(torch.int32)
    assert torch.equal(ops.update_list(u, x), want)


def test_list_checks(cuda):
    from hipims_b200 import ops

    h = torch.ones(10, device=cuda)
    with pytest.raises(RuntimeError, match="CUDA"):
        ops.update_list(h.cpu(), h)
    with pytest.raises(RuntimeError, match="contiguous"):
        ops.update_list(torch.ones(10, 2, device=cuda)[:, 0], h)
    with pytest.raises(RuntimeError, match="dtype"):
        ops.update_list(h.double(), h)
    with pytest.raises(RuntimeError, match="entries"):
        ops.active_list(h, torch.zeros(10, dtype=torch.int32, device=cuda), h[:1])
    assert ops.update_list(h[:0], h[:0]).numel() == 0


@pytest.mark.parametrize("order", [1, 2])
def test_solver_object_equals_the_op_by_op_loop(cuda, order):
    """The native lists against the same loop on an ops object that has only the
    reference's ops: every field, list and clock equal."""
    import types

    from hipims_b200 import ops
    from hipims_b200 import scenarios as S
    from hipims_b200.solver import Godunov

    d = S.urban_catchment(70, seed=4, rain_mm_h=200.0)
    only = types.SimpleNamespace(**{k: getattr(ops, k) for k in (
        "flux_mask", "flux_1st_order", "flux_2nd_order", "friction_update", "update_timestep",
        "station_rain", "device_min")})
    runs = []
    for impl in (None, only):
        g = Godunov(cuda, d["dx"], d["cfl"], 1e9, secondOrder=order == 2, ops_impl=impl)
        mask = torch.as_tensor(d["mask"], device=cuda)
        g.init__fluidField_tensor(mask, d["h"], d["qx"], d["qy"], d["wl"], d["z"], cuda)
        g.set_landuse(mask, d["landuse"], cuda)
        g.set__frictionField_tensor(torch.tensor(d["manning"], dtype=torch.float64), cuda)
        g.set_distributed_rainfall_station_Mask(mask, np.zeros(d["mask"].shape, np.int16), cuda)
        for _ in range(25):
            g.addFlux()
            g.addStation_PrecipitationSource(d["rain"], cuda)
            g.time_friction_euler_update_cuda(cuda)
        runs.append(g)
    a, b = runs
    for f in ("_h_internal", "_qx_internal", "_qy_internal", "_wl_internal", "_h_max", "_wetMask",
              "_accelerator_dt", "t", "dt"):
        assert torch.equal(getattr(a, f), getattr(b, f)), f

"""Arrays and workspaces at the least alignment their elements need, as callers of
the C interface may pass them: the same results as at a torch allocation's."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _records(fs):
    """The solver's host records copied to the device and prepared again."""
    fs.records.copy_(torch.frombuffer(bytearray(fs._recs_host), dtype=torch.uint8))
    fs.prepare()


def _same(a, b):
    x, y = a.compacted(0), b.compacted(0)
    for f in x:
        np.testing.assert_array_equal(x[f], y[f], err_msg=f)
    ca, cb = a.controls()[0], b.controls()[0]
    assert (ca.t, ca.dt, ca.step, ca.status) == (cb.t, cb.dt, cb.step, cb.status)
    assert cb.status == 0


# 8-, 16- and 32-row blocks of the pair step; the FP64 step
@pytest.mark.parametrize("dtype,shape", [(torch.float32, (150, 130)), (torch.float32, (640, 1000)),
                                         (torch.float32, (1200, 1100)),
                                         (torch.float64, (150, 130))])
def test_stations_and_soils_off_their_pair(cuda, dtype, shape):
    from hipims_b200 import scenarios as S
    from hipims_b200.fused import FusedSolver

    rows, cols = shape
    d = S.urban_catchment(cols, n_rows=rows, seed=5, rain_mm_h=150.0)
    rng = np.random.default_rng(1)
    n_st = 7
    rain = np.concatenate([[[0.0] + [1e-5] * n_st], [[1e4] + list(rng.uniform(1e-6, 8e-5, n_st))]])
    c = S.catchment_from(d, rain=rain, rain_station=rng.integers(0, n_st, d["mask"].shape),
                         infiltration=dict(ks=[2e-6, 1e-6], psi=[0.1, 0.2], dtheta=[0.3, 0.2]))
    a, b = (FusedSolver([c], dtype=dtype, device=cuda) for _ in range(2))
    ins = b.inst[0]
    station = torch.zeros(ins.rain_station.numel() + 1, dtype=torch.int16, device=cuda)
    station[1:] = ins.rain_station.view(-1)
    cum = torch.zeros(ins.cum.numel() + 1, dtype=dtype, device=cuda)
    cum[1:] = ins.cum.view(-1)
    b._recs_host[0].rain_station = station.data_ptr() + station.element_size()
    b._recs_host[0].cum = cum.data_ptr() + cum.element_size()
    _records(b)
    for s in (a, b):
        s.step(8)
    ins.cum.copy_(cum[1:].view_as(ins.cum))  # for compacted()
    _same(a, b)
    assert float(ins.cum.max()) > 0.0


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_tile_task_workspace_at_eight_bytes(cuda, dtype):
    from hipims_b200 import scenarios as S
    from hipims_b200.fused import FusedSolver

    c = S.catchment_from(S.urban_catchment(150, n_rows=200, seed=5, rain_mm_h=150.0))
    a, b = (FusedSolver([c], dtype=dtype, device=cuda, kernel="tasks", tile=(32, 32))
            for _ in range(2))
    ws = torch.zeros(b.workspace.numel() + 8, dtype=torch.uint8, device=cuda)
    b.batch.workspace = ws.data_ptr() + 8
    b.prepare()
    for s in (a, b):
        s.step(8)
    _same(a, b)
    assert a.controls()[0].volume == b.controls()[0].volume

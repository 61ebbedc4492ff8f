"""The end of a fused step: rain cursor, boundary-table rows and volume sums of
the clock against the CPU oracle and against plain sums."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _tables(rows, span):
    """Rain, depth, level and discharge tables of `rows` rows over `span` s."""
    t = np.linspace(0.0, span, rows) if rows > 1 else np.zeros(1)
    w = 0.5 + 0.5 * np.sin(np.arange(rows))
    rain = np.stack([t, 2e-5 * (1.0 + w)], 1) if rows > 1 else np.array([[0.0, 1e-5],
                                                                        [span, 1e-5]])
    return (rain, np.stack([t, 0.1 + 0.05 * w], 1), np.stack([t, 0.2 + 0.05 * w], 1),
            np.stack([t, 0.02 * w, 0.01 * w], 1))


# rows around one warp's width; 400 rows over 4 s move the cursor by more than
# a warp's rows in one step (dt grows to about 0.4 s)
@pytest.mark.parametrize("rows", [1, 2, 31, 32, 33, 34, 65, 400])
def test_tables_follow_the_oracle(cuda, rows):
    from hipims_b200 import scenarios as S
    from hipims_b200.fused import FusedSolver
    from oracle.oracle import Sim

    rng = np.random.default_rng(rows)
    mask = np.full((20, 24), 1, dtype=np.int32)
    mask[0, :] = mask[-1, :] = mask[:, 0] = mask[:, -1] = -9999
    mask[1, 1:-1], mask[-2, 1:-1] = 60, 80
    mask[2:-2, 1], mask[2:-2, -2] = 70, 50
    valid = mask > 0
    z = np.where(valid, rng.uniform(0.0, 0.05, mask.shape), 0.0)
    h = np.where(valid, rng.uniform(0.1, 0.2, mask.shape), 0.0)
    rain, gd, gw, gq = _tables(rows, 4.0)
    d = dict(mask=mask, z=z, h=h, qx=np.zeros_like(z), qy=np.zeros_like(z), wl=z + h,
             landuse=np.zeros(mask.shape, np.uint8), manning=[0.03], dx=2.0, cfl=0.5,
             first_dt=0.05, rain=rain, given_depth=gd, given_wl=gw, given_q=gq)
    sim = Sim(d, order=2)
    fs = FusedSolver(S.catchment_from(d), dtype=torch.float64, device=cuda)
    for n in (1, 3, 12):
        sim.step(n)
        fs.step(n)
        c, st = fs.controls()[0], fs.compacted(0)
        # FP64 fused against the oracle: round-off of the one-sided face (1e-10 m)
        assert c.t == pytest.approx(sim.t, rel=1e-9)
        if c.t < rain[-1, 0]:  # the cursor is already at the next step's row
            assert c.rain_index == np.searchsorted(rain[:, 0], c.t, "right") - 1
        for k in ("h", "qx", "qy"):
            np.testing.assert_allclose(st[k], sim.state()[k], rtol=0, atol=1e-10, err_msg=k)


# tiles around the one-level limit of the sums (512 tiles of 32 x 32), and two levels
@pytest.mark.parametrize("shape", [(702, 702), (510, 1022), (520, 1022), (760, 760)])
def test_volume_is_the_sum_of_depths(cuda, shape):
    from hipims_b200 import scenarios as S
    from hipims_b200.fused import FusedSolver

    c = S.catchment_from(S.urban_catchment(shape[1], n_rows=shape[0], seed=5, rain_mm_h=200.0))
    fs = FusedSolver(c, dtype=torch.float64, device=cuda)
    for _ in range(2):
        fs.step(3)
        cc = fs.controls()[0]
        assert cc.volume == pytest.approx(float(fs.compacted(0)["h"].sum()) * c.dx ** 2, rel=1e-12)
        assert cc.volume - cc.volume0 + cc.outflow_volume == pytest.approx(cc.rain_volume, rel=1e-9)


@pytest.mark.parametrize("order", [1, 2])
def test_stations_beyond_the_shared_table(cuda, order):
    """70 stations (more than a tile keeps in shared memory) whose rates repeat
    after 35, against the 35-station form of the same rain: equal bit for bit."""
    from hipims_b200 import scenarios as S
    from hipims_b200.fused import FusedSolver

    d = S.urban_catchment(90, seed=8)
    rng = np.random.default_rng(2)
    rates = rng.uniform(1e-6, 3e-5, (4, 35))
    t = np.array([[0.0], [1.0], [2.5], [1e4]])
    ids = rng.integers(0, 35, d["mask"].shape)
    far = ids + 35 * rng.integers(0, 2, ids.shape)
    runs = []
    for table, st in ((rates, ids), (np.tile(rates, (1, 2)), far)):
        fs = FusedSolver(S.catchment_from(d, rain=np.concatenate([t, table], 1),
                                          rain_station=st), device=cuda, order=order)
        fs.step(30)
        runs.append(fs.compacted(0))
    for k in runs[0]:
        np.testing.assert_array_equal(runs[0][k], runs[1][k], err_msg=k)
    assert runs[0]["h"].max() > 1e-5

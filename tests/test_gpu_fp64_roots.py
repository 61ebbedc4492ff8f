"""The FP64 reciprocal and square root of the step and adjoint kernels
(csrc/hb_fp64.cuh): their stated error bounds against CUDA's correctly rounded
operations, and arguments below the normal range."""
import ctypes
import math
import os
import subprocess

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "chans-hipims-flamegpu_b200")
TINY = np.finfo(np.float64).tiny  # smallest normal number


@pytest.fixture(scope="module")
def check(cuda, tmp_path_factory):
    import build

    out = str(tmp_path_factory.mktemp("fp64") / "libfp64check.so")
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
                    "-shared", "-cudart", "static", "-I", os.path.join(PKG, "csrc"),
                    os.path.join(HERE, "fp64_check.cu"), "-o", out], check=True)
    L = ctypes.CDLL(out)
    L.fp64_check.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]

    def run(x):
        x = torch.as_tensor(x, dtype=torch.float64, device=cuda)
        o = torch.empty(4, x.numel(), dtype=torch.float64, device=cuda)
        assert L.fp64_check(x.numel(), x.data_ptr(), o.data_ptr(),
                            torch.cuda.current_stream(cuda).cuda_stream) == 0
        return o.cpu().numpy()

    return run


# the range the bounds are stated for, its ends' binades, and the whole range in
# which argument and result are normal
@pytest.mark.parametrize("lo,hi", [(-60, 40), (-60, -59), (39, 40), (-1020, 1020)])
def test_error_bounds(check, lo, hi):
    rng = np.random.default_rng(hi - lo)
    x = 2.0 ** rng.integers(lo, hi, 1_000_000) * rng.uniform(1.0, 2.0, 1_000_000)
    x[:4] = 2.0 ** lo, np.nextafter(2.0 ** lo, 4.0), 2.0 ** (hi - 1), 2.0 ** hi * (1 - 2.0 ** -53)
    r, r_ref, s, s_ref = check(x)
    # the stated errors of 2^-53 and 2^-52, and half a unit (2^-53) of the reference
    assert np.max(np.abs(r - r_ref) / r_ref) <= 2.0 ** -52
    assert np.max(np.abs(s - s_ref) / s_ref) <= 2.0 ** -52 + 2.0 ** -53


def test_root_below_the_normal_range(check):
    """Zero, subnormal and negative arguments: a root of zero, as near as the
    root of a subnormal number is to it."""
    x = np.array([0.0, -0.0, 5e-324, 1e-310, np.nextafter(TINY, 0.0), -5e-324, -1.0])
    assert np.array_equal(check(x)[2], np.zeros(7))
    s, ref = check(np.array([TINY, np.nextafter(TINY, 1.0)]))[2:]
    assert np.max(np.abs(s - ref) / ref) <= 2.0 ** -52 + 2.0 ** -53


@pytest.mark.parametrize("order", [1, 2])
def test_depths_that_fade_below_the_normal_range(cuda, order):
    """A Gaussian mound on a flat bed: its tail passes through the subnormal
    numbers to zero, and every cell is active in the first step."""
    from hipims_b200 import scenarios as S
    from hipims_b200.fused import FusedSolver
    from oracle.oracle import Sim

    d = S.dam_break(96)
    valid = d["mask"] > 0
    y, x = np.indices(valid.shape) - 48.0
    d["h"] = np.where(valid, np.exp(-0.35 * (x * x + y * y)), 0.0)
    assert np.any((d["h"] > 0) & (d["h"] < TINY / 9.81))
    d["z"] = np.zeros(valid.shape)
    d["wl"] = d["h"].copy()
    sim = Sim(d, order=order)
    fs = FusedSolver(S.catchment_from(d), dtype=torch.float64, device=cuda, order=order)
    for n in (1, 4):
        sim.step(n)
        fs.step(n)
        got, ref = fs.compacted(0), sim.state()
        assert fs.controls()[0].status == 0
        for f in ("h", "qx", "qy"):
            np.testing.assert_allclose(got[f], ref[f], rtol=0, atol=1e-10, err_msg=f)


@pytest.mark.parametrize("q", [1e-155, 1e-158, 2e-162])
def test_gradient_with_vanishing_discharges(cuda, q):
    """Discharges whose squares are subnormal add nothing to the gradient."""
    from hipims_b200 import scenarios as S
    from hipims_b200.adjoint import GaugeMisfit

    g = []
    for value in (0.0, q):
        mask = np.full((34, 42), -9999, dtype=np.int32)
        mask[1:-1, 1:-1] = 40
        mask[2:-2, 2:-2] = 1
        valid = mask > 0
        d = dict(mask=mask, z=np.zeros(mask.shape), h=np.where(valid, 0.3, 0.0),
                 qx=np.where(valid, value, 0.0), qy=np.where(valid, -value, 0.0),
                 landuse=np.zeros(mask.shape, np.uint8), manning=[0.05], dx=2.0, cfl=0.5,
                 first_dt=0.1, rain=np.array([[0.0, 1e-5], [100.0, 1e-5]]), t_end=math.inf)
        rr, cc = np.nonzero(valid)
        p = GaugeMisfit(S.catchment_from(d), rr, cc, 4, np.full(4, 0.1), every=2,
                        obs=np.zeros((2, rr.size)), device=cuda)
        p.simulate([0.05], 1.0)
        g.append(np.asarray(p.gradient()))
    assert np.all(np.isfinite(g[1]))
    np.testing.assert_allclose(g[1], g[0], rtol=1e-12, atol=1e-15 * np.abs(g[0]).max())

"""Faces of films around the dry depth h_small: at exactly h_small a side is
thin (h <= h_small) but not dry (h < h_small), and the thin side's wave speeds
may cross, or lie on one side of zero with the contact on the other.  There the
reference's two evaluations of a face, one from each cell, differ; the step
kernels evaluate a face once, from its west or south cell, or from the valid
cell of a boundary face."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

HS = 1.0e-6


def _films(n, seed, wall):
    """n x n cells in 2 x 2 blocks of one state (every minmod slope is zero, so the
    edge states are the cells' own in both precisions) on a flat bed, n x n
    inside a one-cell no-data ring, without friction."""
    rng = np.random.default_rng(seed)
    k = n // 2

    def blocks(x):
        return np.pad(np.kron(x, np.ones((2, 2))), 1)

    h = rng.choice([0.0, 5e-7, 9e-7, HS, HS, HS, 4e-5, 9e-5], (k, k))
    u, v = (rng.choice([0.02, 0.2, 1.0], (k, k)) * rng.standard_normal((k, k)) for _ in "uv")
    mask = np.full((n + 2, n + 2), -9999, dtype=np.int32)
    mask[1:-1, 1:-1] = wall
    mask[2:-2, 2:-2] = 1
    return dict(mask=mask, z=np.zeros(mask.shape), h=blocks(h), qx=blocks(h * u),
                qy=blocks(h * v), wl=blocks(h), landuse=np.zeros(mask.shape, np.uint8),
                manning=[0.0], dx=2.0, cfl=0.5, first_dt=0.1)


def _hllc(hL, hR, uL, uR, vL, vR):
    """Mass, normal and tangential momentum flux of a face
    (HC/flucCal_2ndOrder_jh_improved_Kernel.cu:109-195)."""
    g = 9.81
    aL, aR = np.sqrt(g * hL), np.sqrt(g * hR)
    us, as_ = (uL + uR) / 2 + aL - aR, np.abs((aL + aR) / 2 + (uL - uR) / 4)
    sL = np.where(hL <= HS, uR - 2 * aR, np.minimum(uL - aL, us - as_))
    sR = np.where(hR <= HS, uL + 2 * aL, np.maximum(uR + aR, us + as_))
    qL, qR = uL * hL, uR * hR
    nL, nR = uL * qL + g * hL * hL / 2, uR * qR + g * hR * hR / 2
    with np.errstate(all="ignore"):
        sM = (sL * hR * (uR - sR) - sR * hL * (uL - sL)) / (hR * (uR - sR) - hL * (uL - sL))
        hM = (sR * qL - sL * qR + sL * sR * (hR - hL)) / (sR - sL)
        nM = (sR * nL - sL * nR + sL * sR * (qR - qL)) / (sR - sL)
    left = 0 <= sL
    mid_l, mid_r = ~left & (0 <= sM), ~left & (sM < 0) & (0 <= sR)
    wet = ~((hL < HS) & (hR < HS))
    fh = np.where(wet, np.select([left, mid_l | mid_r], [qL, hM], qR), 0.0)
    fn = np.where(wet, np.select([left, mid_l | mid_r], [nL, nM], nR), 0.0)
    return fh, fn, fh * np.where(left | mid_l, vL, vR)


def _one_step(d):
    """h, qx, qy (valid cells) after a step from t = 0 without friction, for states with
    zero slopes on a flat bed in a rectangle with one boundary code."""
    valid = d["mask"] > 0
    kind = int(d["mask"][1, 1]) // 10
    h, qx, qy = d["h"], d["qx"], d["qy"]
    inv = np.where(h < HS, 0.0, 1.0 / np.where(h < HS, 1.0, h))
    u, v = qx * inv, qy * inv
    new = [a.copy() for a in (h, qx, qy)]
    k = d["first_dt"] / d["dx"]
    for axis, (n, t) in enumerate(((u, v), (v, u))):
        def at(a, step):  # the cell `step` along +x, or +y (the row above)
            return np.roll(a, -step, 1) if axis == 0 else np.roll(a, step, 0)

        def ghost(x, normal):
            if kind == 5:
                return x
            flips = axis == 0 if kind == 3 else normal  # RIGID: both on x-faces; SLIP: normal
            return -x if flips else x

        def both(side):  # face between each cell and the next one along side (+1, -1)
            inner = valid & at(valid, side)
            if side > 0:
                f = _hllc(h, at(h, 1), n, at(n, 1), t, at(t, 1))
            else:
                f = _hllc(at(h, -1), h, at(n, -1), n, at(t, -1), t)
            # boundary: from the valid cell, in its outward frame
            b = _hllc(h, h, side * n, side * ghost(n, True), side * t, side * ghost(t, False))
            return [np.where(inner, x, y) for x, y in zip(f, (side * b[0], b[1], b[2]))]

        plus, minus = both(1), both(-1)
        fh, fn, ft = (p - m for p, m in zip(plus, minus))
        new[0] -= k * fh
        new[1 + axis] -= k * fn
        new[2 - axis] -= k * ft
    dry = new[0] < HS
    return [np.where(dry & (i > 0), 0.0, a)[valid] for i, a in enumerate(new)]


# Bounds: dt / dx = 0.05 and four faces a cell.  With depths up to 1e-4 m and
# speeds up to 4 m/s the terms of a face's flux reach 8e-4 (mass) and 5e-3
# (momentum), each good to a few 1e-7 in FP32 and a few 1e-16 in FP64.
TOL = {torch.float32: (5e-10, 3e-9), torch.float64: (1e-17, 1e-16)}


@pytest.mark.parametrize("dtype,wall", [(torch.float32, 30), (torch.float32, 40),
                                        (torch.float32, 50), (torch.float64, 30),
                                        (torch.float64, 40), (torch.float64, 50)])
@pytest.mark.parametrize("order", [1, 2])
def test_films_at_the_dry_depth(cuda, dtype, wall, order):
    from hipims_b200 import scenarios as S
    from hipims_b200.fused import FusedSolver

    tol_h, tol_q = TOL[dtype]
    for seed in range(3):
        d = _films(200, 10 * wall + seed, wall)
        h, qx, qy = _one_step(d)
        fs = FusedSolver(S.catchment_from(d), dtype=dtype, device=cuda, order=order)
        fs.step(1)
        got = fs.compacted(0)
        assert fs.controls()[0].status == 0
        np.testing.assert_allclose(got["h"], h, rtol=0, atol=tol_h, err_msg=f"h {seed}")
        # a film whose fluxes cancel stays at h_small: which side of the dry test its
        # new depth falls on, and so whether it keeps its discharge, is rounding
        sure = np.abs(h - HS) > tol_h
        for f, ref in (("qx", qx), ("qy", qy)):
            np.testing.assert_allclose(got[f][sure], ref[sure], rtol=0, atol=tol_q,
                                       err_msg=f"{f} {seed}")


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_film_moving_off_a_wall(cuda, dtype):
    """A uniform film of exactly h_small that leaves a wall: between the wall's cell
    and its ghost the sides part faster than either can follow."""
    from hipims_b200 import scenarios as S
    from hipims_b200.fused import FusedSolver
    from oracle.oracle import Sim

    d = _films(64, 0, 40)
    valid = d["mask"] > 0
    d["h"] = d["wl"] = np.where(valid, HS, 0.0)
    d["qx"], d["qy"] = np.where(valid, 0.02 * HS, 0.0), np.where(valid, -0.03 * HS, 0.0)
    for order in (1, 2):
        sim = Sim(d, order=order)
        sim.step(1)
        fs = FusedSolver(S.catchment_from(d), dtype=dtype, device=cuda, order=order)
        fs.step(1)
        got, ref = fs.compacted(0), sim.state()
        # depths of 1e-6 and fluxes of 3e-8, the momentum's (g h^2 / 2 within) 5e-12
        tol = 1e-12 if dtype == torch.float32 else 1e-20
        np.testing.assert_allclose(got["h"], ref["h"], rtol=0, atol=tol)
        sure = np.abs(ref["h"] - HS) > tol
        for f in ("qx", "qy"):
            assert np.all(np.isfinite(got[f]))
            np.testing.assert_allclose(got[f][sure], ref[f][sure], rtol=0, atol=tol, err_msg=f)


def test_gradient_through_films(cuda):
    """The adjoint's forward faces (the step's) and its reverse tape on the same
    films, against a central difference in the Manning number."""
    from hipims_b200 import scenarios as S
    from hipims_b200.adjoint import GaugeMisfit

    d = _films(64, 3, 40)
    d["manning"] = [0.02]
    rr, cc = np.nonzero(d["mask"] > 0)
    nsteps = 2  # the Manning number acts on the first step's discharges, so on the depths of the second
    p = GaugeMisfit(S.catchment_from(d), rr, cc, nsteps, np.full(nsteps, 0.1), every=1,
                    checkpoint=2, obs=np.zeros((nsteps, rr.size)), device=cuda,
                    h_reg=-math.inf)

    def J(n):
        return float(p.loss(p.simulate([n], 1.0)))

    J(0.02)
    g = p.gradient()
    assert np.all(np.isfinite(np.asarray(g)))
    eps = 2e-7
    fd = (J(0.02 + eps) - J(0.02 - eps)) / (2 * eps)
    assert float(g[0]) == pytest.approx(fd, rel=1e-3)

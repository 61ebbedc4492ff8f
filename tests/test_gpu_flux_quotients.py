"""The compat flux with the axes' normals (shared slopes and reciprocals) equals
the reference's operation order bit for bit.  The plain form is reached through
normals whose zero components are 1e-300: its products with them vanish against
every operand that is not itself below 1e-290."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TINY = {torch.float64: 1e-300, torch.float32: 1e-36}


def _case(rows, cols, seed, dtype, dev):
    from hipims_b200.topology import compact_index

    rng = np.random.default_rng(seed)
    mask = np.where(rng.uniform(size=(rows, cols)) < 0.9, 10, -9999)
    edge = rng.integers(0, 7, mask.shape)
    mask = np.where(mask > 0, np.choose(edge, [10, 30, 40, 50, 60, 70, 80]), mask)
    mask[0, :] = mask[-1, :] = mask[:, 0] = mask[:, -1] = -9999
    valid = mask > 0
    n = int(valid.sum())
    z = rng.uniform(0.0, 1.0, n) * rng.choice([0.0, 1.0, 30.0], n)
    h = np.choose(rng.integers(0, 5, n), [np.zeros(n), np.full(n, 9e-7), np.full(n, 1.1e-6),
                                          rng.uniform(0, 1e-3, n), rng.uniform(0.1, 3.0, n)])
    q = [np.where(h > 1e-6, h * rng.normal(0, 2.0, n) * rng.choice([0.0, 1e-9, 1.0, 5.0], n), 0.0)
         for _ in range(2)]
    T = lambda x: torch.as_tensor(x, dtype=dtype, device=dev).contiguous()  # noqa: E731
    h, z, qx, qy = T(h), T(z), T(q[0]), T(q[1])
    tabs = [T([[0.0, 0.3], [5.0, 0.4]]), T([[0.0, 0.7]]), T([[0.0, 0.05, -0.02]])]
    return compact_index(torch.as_tensor(mask, device=dev)), h, h + z, z, qx, qy, tabs


def _flux(order, idx, h, wl, z, qx, qy, tabs, normal, dx, dt):
    from hipims_b200 import ops

    n = h.numel()
    out = [torch.full_like(h, 0.1 * (k + 1)) for k in range(3)]
    wet = torch.arange(n, dtype=torch.int32, device=h.device)
    one = lambda v: torch.tensor([v], dtype=h.dtype, device=h.device)  # noqa: E731
    f = ops.flux_2nd_order if order == 2 else ops.flux_1st_order
    f(wet, *out, h, wl, z, qx, qy, idx, normal, *tabs, one(dx), one(1.0), one(dt))
    return torch.stack(out)


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("rows,cols,dx", [(9, 11, 2.0), (120, 133, 0.2012), (64, 300, 3.0)])
def test_axes_equal_the_plain_form(cuda, order, dtype, rows, cols, dx):
    idx, h, wl, z, qx, qy, tabs = _case(rows, cols, rows, dtype, cuda)
    axes = torch.tensor([[1, 0], [0, 1], [-1, 0], [0, -1]], dtype=dtype, device=cuda)
    plain = torch.where(axes == 0, torch.full_like(axes, TINY[dtype]), axes)
    a = _flux(order, idx, h, wl, z, qx, qy, tabs, axes, dx, 0.037)
    b = _flux(order, idx, h, wl, z, qx, qy, tabs, plain, dx, 0.037)
    assert torch.equal(a, b)
    assert float((a - a[:, :1]).abs().max()) > 0


@pytest.mark.parametrize("order", [1, 2])
def test_non_finite_states_follow_the_oracle(cuda, order):
    """Infinite and NaN depths, discharges and beds: the same infinities and NaN
    as the reference's operations, and its values elsewhere."""
    from oracle import oracle as O

    idx, h, wl, z, qx, qy, tabs = _case(40, 50, 3, torch.float64, cuda)
    rng = np.random.default_rng(0)
    for x in (h, qx, qy, z):
        k = torch.as_tensor(rng.choice(h.numel(), 12, replace=False), device=cuda)
        x[k] = torch.tensor([float("inf"), float("-inf"), float("nan")], device=cuda,
                            dtype=x.dtype).repeat(4)
    wl = h + z
    axes = torch.tensor([[1, 0], [0, 1], [-1, 0], [0, -1]], dtype=h.dtype, device=cuda)
    got = _flux(order, idx, h, wl, z, qx, qy, tabs, axes, 2.0, 0.1).cpu().numpy()
    n = h.numel()
    host = lambda t: t.cpu().numpy().copy()  # noqa: E731
    want = [np.full(n, 0.1 * (k + 1)) for k in range(3)]
    O.flux(order, np.arange(n, dtype=np.int32), *want, host(h), host(wl), host(z), host(qx),
           host(qy), host(idx), host(axes).ravel(), *(host(t) for t in tabs), 2.0, 1.0, 0.1)
    want = np.stack(want)
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    assert np.array_equal(np.isnan(got), np.isnan(want))
    # values: cells whose two-cell stencil is finite (next to an infinity or NaN
    # the clamps' choice of a finite operand is the compiler's)
    table = host(idx).reshape(5, n)[1:]
    bad = ~np.isfinite(host(h) + host(z) + host(qx) + host(qy))
    for _ in range(2):
        bad = bad | (np.where(table >= 0, bad[table], False)).any(0)
    assert bad.any() and not bad.all()
    np.testing.assert_allclose(got[:, ~bad], want[:, ~bad], rtol=1e-12, atol=1e-13)

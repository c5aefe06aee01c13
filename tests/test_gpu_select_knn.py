"""GPU parity of select_knn (k nearest neighbours within a radius; the reference's brute-force op
select_knn::select_knn) against the golden vectors of its CPU kernel and the CPU oracle.
Rows are compared as sets (parity.assert_knn_parity): index sets exact up to 1-ulp ties at the
K-th distance, squared distances within 1e-6 relative (measured: bit-identical)."""
import numpy as np
import pytest
import torch

import parity
from oracle import oracle
from test_oracle_pins import load

pytestmark = pytest.mark.gpu

import fastgraphcompute_b200 as fgc  # noqa: E402

DEV = "cuda:0"


def test_golden(golden_dir):
    for name, c in load(golden_dir, "select").items():
        i = c["in"]
        idx, dist = fgc.select_knn(int(i["K"]), torch.as_tensor(i["coords"]).to(DEV),
                                   torch.as_tensor(i["row_splits"]).to(DEV), max_radius=float(i["max_radius"]))
        assert idx.dtype == torch.int64 and dist.dtype == torch.float32
        st = parity.assert_knn_parity(idx.cpu().numpy(), dist.cpu().numpy(), c["out"]["idx"], c["out"]["distsq"],
                                      what=name)
        assert st["max_rel"] == 0.0


def test_random_against_oracle_with_gradient():
    rng = np.random.RandomState(23)
    for trial in range(30):
        sizes = [int(rng.choice([0, 1, rng.randint(2, 30), rng.randint(30, 700)])) for _ in range(rng.randint(1, 5))]
        if sum(sizes) == 0:
            sizes[0] = 6
        rs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
        d = int(rng.randint(2, 6))
        k = int(rng.choice([1, 4, 16, 33, 70]))
        c = rng.rand(int(rs[-1]), d).astype(np.float32)
        r = float(rng.choice([-1.0, 0.05, 0.2, 0.6, 3.0]))
        what = "select case %d (N=%d D=%d K=%d r=%g)" % (trial, c.shape[0], d, k, r)
        coords = torch.as_tensor(c).to(DEV).requires_grad_(True)
        idx, dist = fgc.select_knn(k, coords, torch.as_tensor(rs).to(DEV), max_radius=r)
        oi, od = oracle.select_knn(k, c, rs, r)
        parity.assert_knn_parity(idx.cpu().numpy(), dist.detach().cpu().numpy(), oi, od, what=what)
        if r > 0:
            r2 = np.float32(r * r)
            assert bool((dist.detach().cpu().numpy() <= r2).all())
        up = rng.randn(c.shape[0], k).astype(np.float32)
        (dist * torch.as_tensor(up).to(DEV)).sum().backward()
        og = oracle.binned_select_knn_grad(up, idx.cpu().numpy(), c)
        parity.assert_grad_close(coords.grad.cpu().numpy(), og, what=what + " grad")


def test_radius_filter_entry_point_in_place():
    """fgc_knn_radius_filter on hand-made rows: kept slots close up in order, pads follow."""
    from fastgraphcompute_b200 import _cabi
    idx = torch.tensor([[0, 5, 7, -1, -1], [1, 9, 3, 4, 2], [2, 2, 2, 2, 2]], dtype=torch.int64, device=DEV)
    dist = torch.tensor([[0., 0.5, 0.04, 0., 0.], [0., 0.01, 0.3, 0.02, 0.09], [0., 0., 0., 0., 0.]], device=DEV)
    st = _cabi.current_stream(idx.device)
    a, b = idx[:2].clone(), dist[:2].clone()
    assert _cabi.lib.fgc_knn_radius_filter(_cabi.ptr(a), _cabi.ptr(b), 2, 5, 0.3, 0, st) == 0
    assert a.tolist() == [[0, 7, -1, -1, -1], [1, 9, 4, 2, -1]]
    assert torch.allclose(b, torch.tensor([[0., 0.04, 0., 0., 0.], [0., 0.01, 0.02, 0.09, 0.]], device=DEV))
    a, b = idx.clone(), dist.clone()          # pads written as the point itself
    assert _cabi.lib.fgc_knn_radius_filter(_cabi.ptr(a), _cabi.ptr(b), 3, 5, 0.3, 1, st) == 0
    assert a.tolist() == [[0, 7, 0, 0, 0], [1, 9, 4, 2, 1], [2, 2, 2, 2, 2]]
    a, b = idx.clone(), dist.clone()          # no radius: untouched
    assert _cabi.lib.fgc_knn_radius_filter(_cabi.ptr(a), _cabi.ptr(b), 3, 5, -1.0, 0, st) == 0
    assert torch.equal(a, idx) and torch.equal(b, dist)


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,D,K", [([1], 3, 4), ([0, 2, 0], 2, 3), ([512, 513], 3, 9), ([4096], 4, 17), ([4097, 1], 4, 40), ([16384], 3, 16),
                                       ([16385], 3, 16), ([7] * 600, 3, 5), ([3000, 2000], 6, 20), ([9000, 0, 7000], 4, 66)])
@pytest.mark.parametrize("kind", ["uniform", "clusters"])
@pytest.mark.parametrize("flags", [False, True])
def test_grid_of_a_small_batch(sizes, D, K, kind, flags):
    """The build in one launch and the chain beyond 16384 points: tiles of 4096 threads, row splits beyond those kept in shared memory
    (512), cells of more than 32 and 512 points, four coordinates that fall back to three, direction flags; the same rows twice, and
    the cell order a permutation that the backward may use."""
    import importlib
    import parity
    from oracle import oracle
    km = importlib.import_module("fastgraphcompute_b200.extensions.binned_select_knn")
    g = torch.Generator().manual_seed(sum(sizes) + D)
    n = sum(sizes)
    x = torch.rand((n, D), generator=g)
    if kind == "clusters":
        x = torch.where(torch.rand((n, 1), generator=g) < 0.9, 0.2 + 0.002 * torch.randn((n, D), generator=g), x)
        x[: n // 3] = 0.5
    rs = torch.tensor([0] + sizes).cumsum(0)
    direction = torch.randint(0, 4, (n,), generator=g) if flags else None
    old = km.search_tree
    try:
        km.search_tree = False
        found = [km.knn_forward_with_order(x.cuda(), rs.cuda(), K, None if direction is None else direction.cuda(), False) for _ in range(3)]
    finally:
        km.search_tree = old
    oi, od = oracle.binned_select_knn(K, x.numpy(), rs.numpy(), direction=None if direction is None else direction.numpy())
    for idx, dist, order in found:
        parity.assert_knn_parity(idx.cpu().numpy(), dist.cpu().numpy(), oi, od, what="small grid")
        assert torch.equal(order.long().sort().values.cpu(), torch.arange(n))
    # (D = 4: the first call lets the device choose the form of the grid, the others ask for it)
    assert torch.equal(found[1][0], found[2][0]) and torch.equal(found[1][1], found[2][1]) and torch.equal(found[1][2], found[2][2])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [300, 16384, 20000])
def test_bad_input_of_a_small_batch(n):
    from fastgraphcompute_b200 import binned_select_knn
    x = torch.rand((n, 3), device="cuda")
    x[n - 1, 1] = float("nan")
    with pytest.raises(RuntimeError, match="non-finite"):
        binned_select_knn(5, x, torch.tensor([0, n], device="cuda"))
    x[n - 1, 1] = 0.0
    for bad in ([1, n], [0, n - 1], [0, n, n - 2, n]):
        with pytest.raises(RuntimeError, match="row_splits"):
            binned_select_knn(5, x, torch.tensor(bad, device="cuda"))
    idx, _ = binned_select_knn(5, x, torch.tensor([0, n], device="cuda"))
    assert int(idx.min()) >= 0

"""GPU parity of oc_helper_matrices and select_with_default (the consumers of the same
row_splits data on the loss side) against the reference's known answers, the golden vectors of
its CPU ops, and the CPU oracle on seeded random inputs.  Index work: bit-exact."""
import numpy as np
import pytest
import torch

import parity
from oracle import oracle
from test_oracle_pins import load, OC_KNOWN_ASSO, OC_KNOWN_RS, OC_KNOWN_M, oc_known_m_not

pytestmark = pytest.mark.gpu

import fastgraphcompute_b200 as fgc  # noqa: E402

DEV = "cuda:0"


def run(asso, rs, calc_m_not=True):
    M, M_not, per = fgc.oc_helper_matrices(torch.as_tensor(np.asarray(asso), dtype=torch.int64).to(DEV),
                                           torch.as_tensor(np.asarray(rs), dtype=torch.int64).to(DEV), calc_m_not)
    assert M.dtype == torch.int64 and M_not.dtype == torch.int64 and per.dtype == torch.int64
    assert M.is_cuda and M_not.is_cuda and per.is_cuda
    return M.cpu().numpy(), M_not.cpu().numpy(), per.cpu().numpy()


def test_known_answer_of_the_reference_test():
    """tests/test_oc_helper.py:28-125 of the reference."""
    M, M_not, per = run(OC_KNOWN_ASSO, OC_KNOWN_RS)
    assert M.shape == (7, 4) and M_not.shape == (7, 15)
    parity.assert_oc_matrices_equal(M, M_not, per, OC_KNOWN_M, oc_known_m_not(), [4, 3], "known answer")


def test_golden(golden_dir):
    for name, c in load(golden_dir, "oc").items():
        M, M_not, per = run(c["in"]["asso"], c["in"]["row_splits"])
        parity.assert_oc_matrices_equal(M, M_not, per, c["out"]["M"], c["out"]["M_not"], c["out"]["per_split"], name)
        M2, M_not2, per2 = run(c["in"]["asso"], c["in"]["row_splits"], calc_m_not=False)
        assert np.array_equal(M2, M) and (M_not2 == -1).all() and M_not2.shape == M_not.shape
        assert np.array_equal(per2, per)


def test_random_against_oracle_and_reproducible():
    rng = np.random.RandomState(11)
    for trial in range(25):
        sizes = [int(rng.choice([0, 1, rng.randint(2, 50), rng.randint(50, 3000)])) for _ in range(rng.randint(1, 6))]
        if sum(sizes) == 0:
            sizes[-1] = 7
        rs = np.concatenate([[0], np.cumsum(sizes)])
        hi = int(rng.choice([1, 3, 20, 400]))
        asso = rng.randint(-2, hi, size=int(rs[-1])).astype(np.int64)
        if trial % 4 == 0:
            asso[asso >= 0] *= 2 ** 40 + 3
        a = run(asso, rs)
        b = run(asso, rs)
        for x, y in zip(a, b):
            assert np.array_equal(x, y)          # same rows in the same order on every run
        parity.assert_oc_matrices_equal(*a, *oracle.oc_helper_matrices(asso, rs), "random %d" % trial)
        # rows come ordered by (truth index, row split)
        first = a[0][:, 0] if a[0].shape[1] else np.zeros(0, np.int64)
        keys = [(int(asso[i]), int(np.searchsorted(rs, i, side="right") - 1)) for i in first]
        assert keys == sorted(keys)


def test_edge_cases():
    M, M_not, per = run([-1, -5, -1], [0, 3])               # no object at all
    assert M.shape == (0, 0) and M_not.shape == (0, 3) and per.tolist() == [0]
    M, M_not, per = run([4, 4, 4, 4], [0, 4])                # one object owns its whole row split
    assert M.tolist() == [[0, 1, 2, 3]] and M_not.tolist() == [[-1, -1, -1, -1]] and per.tolist() == [1]
    with pytest.raises(RuntimeError):
        fgc.oc_helper_matrices(torch.zeros(5, dtype=torch.int64, device=DEV),
                               torch.tensor([0, 3], dtype=torch.int64, device=DEV))   # does not end at V
    with pytest.raises(RuntimeError):
        fgc.oc_helper_matrices(torch.zeros(5, dtype=torch.int64), torch.tensor([0, 5]))   # CPU tensors


def test_full_size_properties():
    """16 row splits of 100 000 points, 200 objects each plus noise: every row of M holds exactly the
    points of one (row split, truth index) pair, M_not holds the rest of that row split, ascending."""
    g = torch.Generator().manual_seed(3)
    n_splits, per = 16, 100000
    asso = torch.randint(-20, 200, (n_splits * per,), generator=g)
    rs = torch.arange(0, n_splits * per + 1, per)
    M, M_not, ops = fgc.oc_helper_matrices(asso.to(DEV), rs.to(DEV))
    assert ops.tolist() == [200] * n_splits and M.shape[0] == 200 * n_splits and M_not.shape[1] == per
    ad = asso.to(DEV)
    valid = M >= 0
    first = M[:, 0]
    vals = ad[first]
    # members: same truth index as the first member, same row split, ascending, counts add up
    assert bool(((ad[M.clamp(min=0)] == vals[:, None]) | ~valid).all())
    assert bool((((M // per) == (first // per)[:, None]) | ~valid).all())
    assert bool(((M[:, 1:] > M[:, :-1]) | ~valid[:, 1:]).all())
    assert int(valid.sum()) == int((asso >= 0).sum())
    nvalid = M_not >= 0
    assert bool(((ad[M_not.clamp(min=0)] != vals[:, None]) | ~nvalid).all())
    assert bool((((M_not // per) == (first // per)[:, None]) | ~nvalid).all())
    assert bool(((M_not[:, 1:] > M_not[:, :-1]) | ~nvalid[:, 1:]).all())
    assert bool((valid.sum(1) + nvalid.sum(1) == per).all())


def test_select_with_default_kernel():
    rng = np.random.RandomState(2)
    for dtype, default in ((np.float32, 0.0), (np.float32, -7.5), (np.int64, -1), (np.float64, 2.25), (np.int32, 9)):
        for v, k, f, n in ((50, 7, 3, 50), (200, 16, 1, 120), (33, 4, 32, 64), (0, 5, 3, 10)):
            idx = rng.randint(-1, n, size=(v, k)).astype(np.int64)
            feat = (rng.randn(n, f) * 100).astype(dtype)
            out = fgc.select_with_default(torch.as_tensor(idx).to(DEV), torch.as_tensor(feat).to(DEV), default)
            assert out.shape == (v, k, f) and out.dtype == torch.as_tensor(feat).dtype
            assert np.array_equal(out.cpu().numpy(), oracle.select_with_default(idx, feat, default))
    # the reference's own use: point ids through M (object_condensation.py:148)
    M, _, _ = fgc.oc_helper_matrices(torch.tensor(OC_KNOWN_ASSO, device=DEV), torch.tensor(OC_KNOWN_RS, device=DEV))
    ids = torch.arange(len(OC_KNOWN_ASSO), device=DEV, dtype=torch.int64).view(-1, 1)
    assert torch.equal(fgc.select_with_default(M, ids, -1)[:, :, 0], M)


def test_select_with_default_gradient():
    g = torch.Generator().manual_seed(8)
    idx = torch.randint(-1, 40, (60, 9), generator=g).to(DEV)
    feat = torch.randn((40, 5), generator=g).to(DEV).requires_grad_(True)
    up = torch.randn((60, 9, 5), generator=g).to(DEV)
    (fgc.select_with_default(idx, feat, 0.0) * up).sum().backward()
    ref = torch.zeros((40, 5), dtype=torch.float64)
    ic, uc = idx.cpu(), up.cpu().double()
    for a in range(60):
        for b in range(9):
            if ic[a, b] >= 0:
                ref[ic[a, b]] += uc[a, b]
    parity.assert_grad_close(feat.grad.cpu().numpy(), ref.numpy(), what="select_with_default grad")


@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 40961, 300001])
@pytest.mark.parametrize("kind", ["one byte", "all bytes", "largest", "noise", "one object", "ascending", "gaps"])
def test_sort_of_the_truth_indexes(n, kind):
    """Passes of the sort that are taken and left out, at the edges of its tiles and with more tiles than one look-back reads."""
    rng = np.random.RandomState(n % 1000)
    ids = {"one byte": rng.randint(-3, 200, n), "all bytes": rng.randint(0, 2 ** 62, 300)[rng.randint(0, 300, n)] * 2 + 1,
           "largest": np.where(rng.rand(n) < 0.3, 2 ** 63 - 1, rng.randint(-2, 4, n)), "noise": np.full(n, -1),
           "one object": np.zeros(n), "ascending": np.arange(n) * 255 // n, "gaps": rng.randint(0, 5, n) << 24}[kind].astype(np.int64)
    rs = np.array([0, n // 3, n // 3, n], np.int64)
    M, _, per = run(ids, rs, calc_m_not=False)
    split = (np.arange(n) >= n // 3).astype(np.int64) * 2
    order = np.lexsort((np.arange(n), split, ids))
    order = order[ids[order] >= 0]
    head = np.ones(len(order), bool)
    head[1:] = (ids[order][1:] != ids[order][:-1]) | (split[order][1:] != split[order][:-1])
    rows = np.split(order, np.nonzero(head)[0][1:]) if len(order) else []
    assert M.shape[0] == len(rows) and M.shape[1] == max([len(r) for r in rows], default=0)
    for got, want in zip(M, rows):
        assert np.array_equal(got[:len(want)], want) and (got[len(want):] == -1).all()
    assert np.array_equal(per, [sum(split[r[0]] == e for r in rows) for e in range(3)])


@pytest.mark.parametrize("n", [255, 256, 257, 1023, 1025, 2049, 70002])
@pytest.mark.parametrize("share", [0.002, 0.1, 0.13, 0.5, 0.95])
def test_points_of_no_object(n, share):
    """M_not with few members in the columns that are written at a time, with about as many as the lanes hold, and with more."""
    rng = np.random.RandomState(n)
    ids = np.where(rng.rand(n) < share, 0, 1 + rng.randint(0, 2, n)).astype(np.int64)
    ids[n // 2:n // 2 + n // 8] = 0                                     # members without others between them
    for rs in ([0, n], [0, n // 3, n]):
        M, M_not, _ = run(ids, np.array(rs))
        for k in range(M.shape[0]):
            members = M[k][M[k] >= 0]
            e = np.searchsorted(rs, members[0], side="right") - 1
            want = np.setdiff1d(np.arange(rs[e], rs[e + 1]), members)
            assert np.array_equal(M_not[k][:len(want)], want) and (M_not[k][len(want):] == -1).all()


@pytest.mark.parametrize("n", [4097, 300001])
def test_a_status_ends_every_pass_of_the_sort(n):
    """A status that is set when the passes begin: all CTAs of all of them leave, and nothing is kept from it for the next call."""
    ids = (torch.arange(n, device=DEV) % 40) << 20
    for _ in range(3):
        with pytest.raises(RuntimeError, match="row_splits"):
            fgc.oc_helper_matrices(ids, torch.tensor([0, n, n - 1, n], device=DEV))
        M, _, per = run(ids.cpu(), [0, n], calc_m_not=False)
        assert M.shape[0] == 40 == per[0] and np.array_equal(M[:, 0], np.arange(40))


@pytest.mark.parametrize("n_maxrs", [0x7fffffff, 0x7ffffffe, 0x7fffff01])
def test_columns_up_to_31_bits(n_maxrs):
    """Rows as long as fgc_oc_fill takes them: the last steps reach beyond 31 bits.  Nothing before or behind the row is written."""
    import ctypes
    from fastgraphcompute_b200 import _cabi
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 17 GB")
    lib, ptr = _cabi.lib, _cabi.ptr
    asso, rs = torch.tensor([-1, 3, -1, 3, -1], device=DEV), torch.tensor([0, 5], device=DEV)
    nbytes, stream = lib.fgc_oc_workspace_bytes(5), _cabi.current_stream(asso.device)
    ws, per = torch.empty(nbytes, dtype=torch.uint8, device=DEV), torch.empty(1, dtype=torch.int64, device=DEV)
    assert lib.fgc_oc_prepare(ptr(asso), 5, ptr(rs), 2, ptr(ws), nbytes, ptr(per), stream) == 0
    status, sizes = ctypes.c_int32(0), (ctypes.c_int64 * 3)()
    assert lib.fgc_oc_read_sizes(ptr(ws), ctypes.byref(status), sizes, stream) == 0 and list(sizes) == [1, 2, 5]
    M = torch.empty((1, 2), dtype=torch.int64, device=DEV)
    room = torch.full((n_maxrs + 64,), -7, dtype=torch.int64, device=DEV)
    row = room[32:32 + n_maxrs]
    assert lib.fgc_oc_fill(ptr(ws), nbytes, 5, ptr(rs), 1, 2, n_maxrs, ptr(M), ptr(row), stream) == 0
    assert M.tolist() == [[1, 3]] and row[:4].tolist() == [0, 2, 4, -1]
    assert (room[:32] == -7).all() and (room[32 + n_maxrs:] == -7).all()
    for part in row[3:].split(1 << 28):
        assert int(part.min()) == -1 == int(part.max())


def test_an_internal_status_is_an_error(monkeypatch):
    """(a sort that gave up leaves no objects, which would look like a result)"""
    from fastgraphcompute_b200 import _cabi
    read = _cabi.lib.fgc_oc_read_sizes

    def gave_up(ws, status, sizes, stream):
        rc = read(ws, status, sizes, stream)
        status._obj.value |= _cabi.STATUS_INTERNAL
        return rc
    monkeypatch.setattr(_cabi.lib, "fgc_oc_read_sizes", gave_up)
    with pytest.raises(RuntimeError, match="status 32"):
        fgc.oc_helper_matrices(torch.zeros(5, dtype=torch.int64, device=DEV), torch.tensor([0, 5], device=DEV))

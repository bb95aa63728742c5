"""Tensor-core histograms (te_mma.cu) against the oracle and against the
shared-memory kernel, which takes every pair when the workspace has no room for the
tensor-core path's tables and bit planes.

Counts are whole numbers and compared exactly. TE: both kernels evaluate the same
float32 expression per cell and differ in the order of the sums; a term's rounding is
at most 2^-23 of its count, so two sums of N counts differ by less than 1e-6 per
sample."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tenex_b200 import native
from tenex_b200.kernels import device as D

pytestmark = pytest.mark.gpu
TOL = 1e-6


def _bins(seed, n, T, b_lo, b_hi, K=1, skew=False):
    rng = np.random.default_rng(seed)
    b = rng.integers(b_lo, b_hi + 1, n)
    x = np.stack([rng.integers(0, v, T * K) for v in b])
    if skew:  # rare bins: target states that never occur, empty (xt, y) columns
        x = np.where(rng.random(x.shape) < 0.8, 0, x)
    bins, npv, bmax = O.remap(x.astype(np.int32))
    return bins.reshape(n, T, K), npv, bmax


def _run(db, npv, bmax, lag, p0, cnt, dev, tensor_cores, matrix=False, counts=None):
    """(TE, raw counts) of pair ids [p0, p0 + cnt) through the C ABI; tensor_cores =
    False gives the call the workspace of the shared-memory kernel only."""
    full = D.workspace(dev, db.n, db.row_len, bmax)
    ws = full if tensor_cores else D.workspace(dev, db.n, db.row_len, bmax, pair_list=True)
    out = torch.zeros((db.n, db.n) if matrix else cnt, dtype=torch.float32, device=dev)
    s = native.stream_ptr()
    if counts is None:
        native.call("tenex_te_pairfree", db.ptr(), db.ld, npv.data_ptr(), bmax, db.n, db.row_len,
                    lag, p0, cnt, out.data_ptr(),
                    native.OUT_MATRIX if matrix else native.OUT_PAIRFREE, db.n if matrix else 0,
                    ws.data_ptr(), ws.numel(), None, s)
    else:
        native.call("tenex_te_pairfree_counts", db.ptr(), db.ld, npv.data_ptr(), bmax, db.n,
                    db.row_len, lag, p0, cnt, out.data_ptr(), counts.data_ptr(), bmax ** 3,
                    ws.data_ptr(), ws.numel(), None, s)
    native.call("tenex_workspace_status", ws.data_ptr(), s)
    return out


# (genes, samples, bins, lag): one gene pair; sample counts around the 64-sample MMA,
# the 256-sample step and the ring of stages; lags past a word and past a step; bins
# around the largest target (16), rows that fill a tile unevenly, wide sources
SHAPES = [(2, 2, (1, 3), 1), (3, 65, (2, 4), 1), (9, 256, (2, 2), 1), (9, 257, (2, 5), 1),
          (12, 320, (3, 7), 33), (40, 769, (2, 9), 1), (150, 511, (1, 2), 1),
          (70, 1030, (2, 16), 3), (60, 1500, (13, 16), 1), (30, 2049, (2, 38), 300),
          (25, 700, (5, 38), 1), (131, 1024, (4, 4), 1)]


@pytest.mark.parametrize("n,T,b,lag", SHAPES)
@pytest.mark.parametrize("skew", [False, True])
def test_counts_and_te(cuda, n, T, b, lag, skew):
    bins, npv, bmax = _bins(n * T + skew, n, T, *b, skew=skew)
    db = D.pack_bins(bins, cuda)
    npv_t = torch.as_tensor(npv, dtype=torch.int32, device=cuda)
    P = n * (n - 1)
    ref = O.te_pairfree(bins, npv, tau=lag)
    lo, hi = (P // 3, P - P // 5) if P > 6 else (0, P)   # a range that cuts targets
    te = [_run(db, npv_t, bmax, lag, 0, P, cuda, tc).cpu().numpy() for tc in (True, False)]
    assert np.max(np.abs(te[0] - ref)) <= TOL
    assert np.max(np.abs(te[0] - te[1])) <= TOL
    part = _run(db, npv_t, bmax, lag, lo, hi - lo, cuda, True).cpu().numpy()
    # a pair's value does not depend on the range, so not on its tile
    few = (bmax ** 3 <= 1200)
    assert np.max(np.abs(part - te[0][lo:hi])) <= (0 if few else TOL)
    m = _run(db, npv_t, bmax, lag, 0, P, cuda, True, matrix=True).cpu().numpy()
    assert np.array_equal(m.T[~np.eye(n, dtype=bool)], te[0]) and not m.diagonal().any()
    if P * bmax ** 3 <= 40_000_000:
        c = [torch.full((P, bmax ** 3), -1, dtype=torch.int32, device=cuda) for _ in range(2)]
        t = [_run(db, npv_t, bmax, lag, 0, P, cuda, tc, counts=k).cpu().numpy()
             for tc, k in zip((True, False), c)]
        assert torch.equal(c[0], c[1])
        assert np.array_equal(t[0], te[0])


def test_counts_exact_up_to_2_pow_24(cuda):
    """float32 accumulators hold every count of the longest series the path takes:
    constant genes give one cell of all N samples."""
    T = (1 << 24) - 3
    rng = np.random.default_rng(7)
    x = np.zeros((4, T), np.uint8)
    x[1] = rng.random(T) < 1e-6
    x[2] = rng.random(T) < 0.5
    x[1, 5], x[2, 9], x[3] = 1, 1, 1 - x[1]
    npv = np.array([1, 2, 2, 2], np.int32)
    db = D.pack_bins(x, cuda)
    npv_t = torch.as_tensor(npv, device=cuda)
    c = [torch.zeros((12, 8), dtype=torch.int32, device=cuda) for _ in range(2)]
    te = [_run(db, npv_t, 2, 1, 0, 12, cuda, tc, counts=k) for tc, k in zip((True, False), c)]
    assert torch.equal(c[0], c[1])
    assert float((te[0] - te[1]).abs().max()) <= TOL


def test_kernel_dimension_and_surrogate_statistics(cuda):
    bins, npv, bmax = _bins(3, 45, 400, 2, 8, K=2)
    db = D.pack_bins(bins, cuda)
    npv_t = torch.as_tensor(npv, dtype=torch.int32, device=cuda)
    te = D.te_pairfree(db, npv_t, bmax, 2, matrix=True)
    ref = _run(db, npv_t, bmax, 4, 0, 45 * 44, cuda, False, matrix=True)
    assert float((te - ref).abs().max()) <= TOL
    obs = torch.full((45, 45), float(te.median()), device=cuda)
    acc = [torch.zeros((45, 45), dtype=torch.float64, device=cuda) for _ in range(2)]
    cnt = torch.zeros((45, 45), dtype=torch.int32, device=cuda)
    for _ in range(2):
        D.surrogate_accumulate(db, npv_t, bmax, 2, obs, acc[0], acc[1], cnt)
    off = ~torch.eye(45, dtype=torch.bool, device=cuda)
    assert torch.equal(acc[0], 2 * te.double())
    assert torch.equal(acc[1], 2 * te.double() ** 2)
    assert torch.equal(cnt[off], 2 * (te >= obs).int()[off])
    assert not cnt[~off].any()


@pytest.mark.parametrize("low", [0, 7, 13])
def test_targets_that_use_few_of_their_bins(cuda, low):
    """Targets of 16 bins whose values lie in three of them: one of the two halves that
    the epilogue splits a target's bins into has no columns (low 0, 13) or both have."""
    rng = np.random.default_rng(low)
    n, T = 30, 700
    bins = rng.integers(0, 3, (n, T)).astype(np.uint8)
    npv = np.full(n, 3, np.int32)
    bins[::2] += np.uint8(low)
    npv[::2] = 16
    db = D.pack_bins(bins, cuda)
    npv_t = torch.as_tensor(npv, dtype=torch.int32, device=cuda)
    P = n * (n - 1)
    te = [_run(db, npv_t, 16, 1, 0, P, cuda, tc).cpu().numpy() for tc in (True, False)]
    assert np.max(np.abs(te[0] - O.te_pairfree(bins, npv, tau=1))) <= TOL
    assert np.max(np.abs(te[0] - te[1])) <= TOL


def _all_outputs_match_oracle(bins, npv, bmax, lag, dev):
    """Pair-free and matrix output and surrogate statistics of every pair, with the
    tensor-core path, against the oracle. The value of N samples is a mean of N terms, so
    TOL per sample holds for short series as for long ones."""
    n = len(npv)
    P, off = n * (n - 1), ~np.eye(n, dtype=bool)
    db = D.pack_bins(bins, dev)
    npv_t = torch.as_tensor(npv, dtype=torch.int32, device=dev)
    ref = O.te_pairfree(bins, npv, tau=lag)
    te = _run(db, npv_t, bmax, lag, 0, P, dev, True)
    assert np.max(np.abs(te.cpu().numpy() - ref)) <= TOL
    m = _run(db, npv_t, bmax, lag, 0, P, dev, True, matrix=True)
    assert np.array_equal(m.cpu().numpy().T[off], te.cpu().numpy())
    acc = [torch.zeros((n, n), dtype=torch.float64, device=dev) for _ in range(2)]
    cnt = torch.zeros((n, n), dtype=torch.int32, device=dev)
    D.surrogate_accumulate(db, npv_t, bmax, lag, m, acc[0], acc[1], cnt)
    assert torch.equal(acc[0], m.double()) and torch.equal(acc[1], m.double() ** 2)
    assert np.array_equal(cnt.cpu().numpy(), off.astype(np.int32))


@pytest.mark.parametrize("wide", [0, 1, 6])
def test_targets_of_many_bins_and_few_states(cuda, wide):
    """Targets of 8 to 16 declared bins that use one or two of them (1 to 4 occupied
    states): both low, both high, one of each half; beside each other in a tile and, with
    `wide`, beside targets of many states."""
    rng = np.random.default_rng(40 + wide)
    T, rows, npv = 400, [], []
    for b in (8, 9, 11, 16) * 10:
        for v0, v1 in ((0, 0), (b - 1, b - 1), (0, 1), (b - 2, b - 1), (0, b - 1), (b // 2, 1)):
            rows.append(np.where(rng.random(T) < 0.4, v0, v1))
            npv.append(b)
        rows.append(np.r_[np.zeros(T - 1, np.int64), b - 1])   # its second value comes last
        npv.append(b)
    for i in range(5 + wide):
        b = 2 + i if i < 5 else 16
        rows.append(rng.integers(0, b, T))
        npv.append(b)
    order = rng.permutation(len(rows))
    bins = np.stack(rows)[order].astype(np.uint8)
    _all_outputs_match_oracle(bins, np.array(npv, np.int32)[order], 16, 1, cuda)


@pytest.mark.parametrize("T,lag", [(2, 1), (12, 6), (20, 15), (33, 31), (60, 50), (60, 53),
                                   (300, 292)])
def test_lag_close_to_the_length(cuda, T, lag):
    """Dense genes of 8 to 16 bins with T - lag from 1 to 10: fewer samples than bins."""
    bins, npv, bmax = _bins(1000 * T + lag, 250, T, 8, 16)
    _all_outputs_match_oracle(bins[:, :, 0].astype(np.uint8), npv, bmax, lag, cuda)


@pytest.mark.parametrize("T,tau", [(40, 39), (60, 54), (120, 111)])
def test_engine_with_a_lag_close_to_the_length(cuda, T, tau):
    from tenex_b200 import TransferEntropyEngine
    rng = np.random.default_rng(T)
    x = np.log1p(rng.poisson(3.0, (240, T)) * (rng.random((240, T)) < 0.7)).astype(np.float32)
    res = TransferEntropyEngine(x, np.array([f"g{i}" for i in range(240)])).compute(
        accelerator="gpu", tau=tau, kp=0.5)
    ref = O.te_matrix(np.asarray(res.bin_arrs), np.asarray(res.n_per_var), tau=tau)
    assert np.max(np.abs(res.matrix - ref)) <= TOL


@pytest.mark.parametrize("offset", [4, 8, 20, 128, 252])
def test_workspace_at_any_word(cuda, offset):
    """The entry points accept a workspace at any multiple of 4 bytes: the tensor-core
    tables start at the next multiple of 256 bytes in it, in a smaller part of it."""
    bins, npv, bmax = _bins(offset, 300, 900, 2, 16)
    db = D.pack_bins(bins, cuda)
    npv_t = torch.as_tensor(npv, dtype=torch.int32, device=cuda)
    P, s = 300 * 299, native.stream_ptr()
    out = torch.zeros(P, dtype=torch.float32, device=cuda)
    nb = D.workspace(cuda, 300, db.row_len, bmax).numel()
    mem = torch.full((nb + 512,), 85, dtype=torch.uint8, device=cuda)
    ws = mem[offset:offset + nb]
    native.call("tenex_te_pairfree", db.ptr(), db.ld, npv_t.data_ptr(), bmax, 300, db.row_len, 1,
                0, P, out.data_ptr(), native.OUT_PAIRFREE, 0, ws.data_ptr(), nb, None, s)
    native.call("tenex_workspace_status", ws.data_ptr(), s)
    assert np.max(np.abs(out.cpu().numpy() - O.te_pairfree(bins, npv, tau=1))) <= TOL
    assert bool((mem[:offset] == 85).all()) and bool((mem[offset + nb:] == 85).all())


@pytest.mark.parametrize("b_hi", [7, 16, 38])
@pytest.mark.parametrize("part", [0.02, 0.3, 0.55, 0.9])
def test_workspace_with_room_for_some_genes(cuda, b_hi, part):
    """Between the least and the full workspace the bit planes reach only some of the
    sources, cut inside a class of one bin count; the other pairs run in the
    shared-memory kernel."""
    bins, npv, bmax = _bins(b_hi, 300, 800, 2, b_hi)
    db = D.pack_bins(bins, cuda)
    npv_t = torch.as_tensor(npv, dtype=torch.int32, device=cuda)
    P, s = 300 * 299, native.stream_ptr()
    out = torch.zeros(P, dtype=torch.float32, device=cuda)
    full = D.workspace(cuda, 300, db.row_len, bmax).numel()
    planes = 300 * min(bmax, 16) * (1024 // 8 * 2)          # the part that holds bit planes
    nb = full - int(planes * (1 - part)) // 4 * 4
    ws = torch.empty(nb, dtype=torch.uint8, device=cuda)
    native.call("tenex_te_pairfree", db.ptr(), db.ld, npv_t.data_ptr(), bmax, 300, db.row_len, 1,
                0, P, out.data_ptr(), native.OUT_PAIRFREE, 0, ws.data_ptr(), nb, None, s)
    native.call("tenex_workspace_status", ws.data_ptr(), s)
    assert np.max(np.abs(out.cpu().numpy() - O.te_pairfree(bins, npv, tau=1))) <= TOL


@pytest.mark.parametrize("bt,bs", [(15, 3), (13, 8), (7, 2)])
def test_error_is_no_larger_than_the_counting_kernels(cuda, bt, bs):
    """Root mean square error against the float64 oracle on short series, where TE and so
    the sums are large. Both kernels add float32 terms in chains of a column or so and the
    rest in float64, so their errors have one size; 10% is left for the 1% by which the
    root mean square of 19,600 errors varies and the terms' order."""
    n, T = 280, 300
    rng = np.random.default_rng(bt)
    bins, npv, bmax = O.remap(np.stack(
        [rng.integers(0, bt if i % 2 else bs, T) for i in range(n)]).astype(np.int32))
    db = D.pack_bins(bins, cuda)
    npv_t = torch.as_tensor(npv, dtype=torch.int32, device=cuda)
    P = n * (n - 1)
    ids = np.arange(P)
    tgt, src = ids // (n - 1), ids % (n - 1)
    mine = (npv[tgt] == bt) & (npv[src + (src >= tgt)] == bs)
    ref = O.te_pairfree(bins, npv, tau=1)
    rms = [float(np.sqrt(np.mean((_run(db, npv_t, bmax, 1, 0, P, cuda, tc).cpu().numpy().astype(
        np.float64) - ref)[mine] ** 2))) for tc in (True, False)]
    assert mine.sum() == 140 * 140 and rms[0] <= 1.1 * rms[1]


@pytest.mark.parametrize("n,T,b", [(260, 300, (2, 16)), (300, 1200, (2, 12)),
                                   (340, 2000, (2, 38)), (230, 70000, (2, 24))])
def test_value_of_a_pair_is_the_same_by_every_route(cuda, n, T, b):
    """Tensor cores or shared-memory counters of 32 or 16 bits, any launch shape, pair range
    or list: the terms of a column are added in one order in float32, all else in
    float64, whose order leaves a float32 result of these inputs alone."""
    from tenex_b200.kernels.pair_list import te_pair_list
    bins, npv, bmax = _bins(n + T, n, T, *b, skew=True)
    db = D.pack_bins(bins, cuda)
    npv_t = torch.as_tensor(npv, dtype=torch.int32, device=cuda)
    P = n * (n - 1)
    te = _run(db, npv_t, bmax, 1, 0, P, cuda, True)
    assert torch.equal(te, _run(db, npv_t, bmax, 1, 0, P, cuda, False))
    for p0, cnt in ((0, 50), (P // 2 - 7, 3 * n), (P - n, n)):
        for tc in (True, False):
            assert torch.equal(te[p0:p0 + cnt], _run(db, npv_t, bmax, 1, p0, cnt, cuda, tc))
    for cfg in (dict(threads=1024, ctas_per_sm=1, src_chunk=512),
                dict(threads=256, ctas_per_sm=2, src_chunk=64),
                dict(threads=128, ctas_per_sm=4, src_chunk=7)):
        assert torch.equal(te, D.te_pairfree(db, npv_t, bmax, 1, cfg=cfg))
    ids = np.random.default_rng(n).integers(0, P, 2000)
    tgt, loc = ids // (n - 1), ids % (n - 1)
    pl = te_pair_list(db, npv_t, bmax, 1, np.stack((tgt, loc + (loc >= tgt)), 1))
    assert torch.equal(te[torch.as_tensor(ids, device=cuda)], pl)


def _items(ws):
    """Work items of the tensor-core launch that used this workspace (0: there was none)."""
    return int(ws[16:20].view(torch.int32))


# the edges of SHAPES, with the genes that make the tensor-core path worth its launches
@pytest.mark.parametrize("n,T,b,lag", [
    (230, 2, (1, 3), 1), (230, 65, (2, 4), 1), (230, 256, (2, 2), 1), (230, 257, (2, 5), 1),
    (231, 320, (3, 7), 33), (240, 769, (2, 9), 1), (231, 1024, (4, 4), 1),
    (330, 1030, (2, 16), 3), (340, 1500, (13, 16), 1), (360, 2049, (2, 38), 300),
    (300, 700, (5, 38), 1)])
@pytest.mark.parametrize("skew", [False, True])
def test_counts_and_te_of_enough_genes(cuda, n, T, b, lag, skew):
    bins, npv, bmax = _bins(n * T + skew, n, T, *b, skew=skew)
    bmax = max(bmax, b[1])            # declared, so that the size decides and not the draw
    db = D.pack_bins(bins, cuda)
    npv_t = torch.as_tensor(npv, dtype=torch.int32, device=cuda)
    P, s = n * (n - 1), native.stream_ptr()
    ref = O.te_pairfree(bins, npv, tau=lag)
    ws = D.workspace(cuda, n, db.row_len, bmax)
    m = torch.zeros((n, n), dtype=torch.float32, device=cuda)
    native.call("tenex_te_pairfree", db.ptr(), db.ld, npv_t.data_ptr(), bmax, n, db.row_len, lag,
                0, P, m.data_ptr(), native.OUT_MATRIX, n, ws.data_ptr(), ws.numel(), None, s)
    native.call("tenex_workspace_status", ws.data_ptr(), s)
    assert _items(ws) > 0 and not bool(m.diagonal().any())
    te = _run(db, npv_t, bmax, lag, 0, P, cuda, True).cpu().numpy()
    assert np.max(np.abs(te - ref)) <= TOL
    assert np.array_equal(m.cpu().numpy().T[~np.eye(n, dtype=bool)], te)
    for p0, cnt in ((P // 9, P - P // 5), (P // 2, n // 2)):  # ranges that cut targets
        part = _run(db, npv_t, bmax, lag, p0, cnt, cuda, True).cpu().numpy()
        assert np.array_equal(part, te[p0:p0 + cnt])
    if P * bmax ** 3 <= 60_000_000:
        c = [torch.full((P, bmax ** 3), -1, dtype=torch.int32, device=cuda) for _ in range(2)]
        t = [_run(db, npv_t, bmax, lag, 0, P, cuda, tc, counts=k).cpu().numpy()
             for tc, k in zip((True, False), c)]
        assert torch.equal(c[0], c[1])
        assert np.array_equal(t[0], te) and np.array_equal(t[1], te)


def test_counts_of_tensor_cores_exact_up_to_2_pow_24(cuda):
    """float32 accumulators hold every count of the longest series the path takes; twenty
    genes of it are enough work."""
    T, n = (1 << 24) - 3, 20
    rng = np.random.default_rng(8)
    x = np.zeros((n, T), np.uint8)
    for i in range(1, n):
        x[i] = rng.random(T) < (0.5, 1e-6, 1 - 1e-6)[i % 3]
        x[i, i], x[i, i + 20] = 0, 1
    npv = np.array([1] + [2] * (n - 1), np.int32)
    db = D.pack_bins(x, cuda)
    npv_t = torch.as_tensor(npv, device=cuda)
    P = n * (n - 1)
    c = [torch.zeros((P, 8), dtype=torch.int32, device=cuda) for _ in range(2)]
    te = [_run(db, npv_t, 2, 1, 0, P, cuda, tc, counts=k) for tc, k in zip((True, False), c)]
    assert D.workspace(cuda, n, db.row_len, 2).numel() > n * T // 2   # with room for planes
    assert torch.equal(c[0], c[1]) and int(c[0].sum(1).min()) == T - 1
    assert float((te[0] - te[1]).abs().max()) <= TOL


def test_small_launches_run_without_the_tensor_cores(cuda):
    """Few genes and ranges of few pairs go to the counting kernel alone (its ticket says
    so: no work item of the other path), which is the faster there, with equal results."""
    for n, T, b, cnt in ((40, 2000, (2, 6), None), (10, 60_000, (2, 16), None),
                         (800, 3000, (2, 16), 300)):
        bins, npv, bmax = _bins(n, n, T, *b)
        db = D.pack_bins(bins, cuda)
        npv_t = torch.as_tensor(npv, dtype=torch.int32, device=cuda)
        P = n * (n - 1) if cnt is None else cnt
        ws = torch.empty(64 << 20, dtype=torch.uint8, device=cuda)
        out = torch.zeros(P, dtype=torch.float32, device=cuda)
        native.call("tenex_te_pairfree", db.ptr(), db.ld, npv_t.data_ptr(), bmax, n, db.row_len,
                    1, 0, P, out.data_ptr(), native.OUT_PAIRFREE, 0, ws.data_ptr(), ws.numel(),
                    None, native.stream_ptr())
        assert _items(ws) == 0
        ref = O.te_pairfree(bins, npv, 1, 0, P)
        assert np.max(np.abs(out.cpu().numpy() - ref)) <= TOL


@pytest.mark.parametrize("b_hi", [7, 16, 38])
@pytest.mark.parametrize("part,taken", [(0.02, False), (0.3, True), (0.55, True), (0.9, True)])
def test_part_of_the_workspace_is_used_where_it_is_worth_it(cuda, b_hi, part, taken):
    """Room for a few genes' bit planes only: the path's launches take longer than they
    save, so the counting kernel runs alone; with room for more the planes are cut inside a
    class of one bin count."""
    n, T = 500, 1200
    bins, npv, bmax = _bins(b_hi + 1, n, T, 2, b_hi)
    bmax = max(bmax, b_hi)
    db = D.pack_bins(bins, cuda)
    npv_t = torch.as_tensor(npv, dtype=torch.int32, device=cuda)
    P, s = n * (n - 1), native.stream_ptr()
    out = torch.zeros(P, dtype=torch.float32, device=cuda)
    planes = n * min(bmax, 16) * (1280 // 8 * 2)            # the part that holds bit planes
    nb = D.workspace(cuda, n, db.row_len, bmax).numel() - int(planes * (1 - part)) // 4 * 4
    ws = torch.empty(nb, dtype=torch.uint8, device=cuda)
    native.call("tenex_te_pairfree", db.ptr(), db.ld, npv_t.data_ptr(), bmax, n, db.row_len, 1,
                0, P, out.data_ptr(), native.OUT_PAIRFREE, 0, ws.data_ptr(), nb, None, s)
    native.call("tenex_workspace_status", ws.data_ptr(), s)
    assert (_items(ws) > 0) == taken
    assert np.max(np.abs(out.cpu().numpy() - O.te_pairfree(bins, npv, tau=1))) <= TOL


def test_captured_launch_and_two_streams(cuda):
    """The tensor-core path in a CUDA graph replayed on other bins, and from two threads with
    a stream and a workspace each: the values of an eager call."""
    import threading
    n, T, lag = 320, 1100, 1
    sets = [_bins(seed, n, T, 2, 12) for seed in (1, 2)]
    bmax = 12
    dbs = [D.pack_bins(b, cuda) for b, _, _ in sets]
    npvs = [torch.as_tensor(p, dtype=torch.int32, device=cuda) for _, p, _ in sets]
    P = n * (n - 1)
    want = [_run(d, p, bmax, lag, 0, P, cuda, True) for d, p in zip(dbs, npvs)]
    assert not torch.equal(want[0], want[1])

    def call(db, npv, out, ws):
        native.call("tenex_te_pairfree", db.ptr(), db.ld, npv.data_ptr(), bmax, n, db.row_len,
                    lag, 0, P, out.data_ptr(), native.OUT_PAIRFREE, 0, ws.data_ptr(), ws.numel(),
                    None, native.stream_ptr())

    ws = D.workspace(cuda, n, dbs[0].row_len, bmax)
    db, npv, out = D.pack_bins(sets[0][0], cuda), npvs[0].clone(), torch.zeros_like(want[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(db, npv, out, ws)
    for k in (0, 1, 0):
        db.data.copy_(dbs[k].data)
        npv.copy_(npvs[k])
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert _items(ws) > 0 and torch.equal(out, want[k])

    got = [torch.zeros_like(w) for w in want]
    failed = []

    def work(k):
        try:
            torch.cuda.set_device(cuda)
            s = torch.cuda.Stream(cuda)
            with torch.cuda.stream(s):
                mine = D.workspace(cuda, n, dbs[k].row_len, bmax)
                for _ in range(20):
                    call(dbs[k], npvs[k], got[k], mine)
                native.call("tenex_workspace_status", mine.data_ptr(), native.stream_ptr())
            s.synchronize()
        except Exception as e:  # shown by the assertion below
            failed.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed and all(torch.equal(g, w) for g, w in zip(got, want))

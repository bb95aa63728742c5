"""Host-side parts of the device layer that need no GPU."""
import os
import threading

import numpy as np
import pytest
import torch

from tenex_b200 import native
from tenex_b200.kernels import device as D


def test_to_device_takes_a_tensor_that_requires_grad():
    x = torch.arange(6, dtype=torch.float32).reshape(2, 3)
    got = D.to_device(x.clone().requires_grad_(), "cpu")
    assert torch.equal(got, x)


def test_workspace_falls_back_to_the_least_when_memory_is_short(monkeypatch):
    L = native.lib()
    full = L.tenex_te_workspace_bytes(1000, 3000, 16)
    least = L.tenex_te_pairs_workspace_bytes(1000, 3000, 16)
    assert full > least
    real, asked = torch.empty, []

    def empty(nb, **kw):
        asked.append(nb)
        if nb > least:
            raise torch.OutOfMemoryError("no room")
        return real(nb, **kw)

    monkeypatch.setattr(torch, "empty", empty)
    assert D.workspace("cpu", 1000, 3000, 16).numel() == least and asked == [full, least]
    monkeypatch.setattr(torch, "empty", lambda *a, **k: (_ for _ in ()).throw(
        torch.OutOfMemoryError("no room")))
    with pytest.raises(torch.OutOfMemoryError):
        D.workspace("cpu", 1000, 3000, 16)


def test_workspace_of_small_problems_is_the_least():
    """Few genes, whatever the series' length, run without the tensor-core path: their
    workspace holds none of its tables and planes."""
    L = native.lib()
    for n, T, b in ((2, 2, 2), (2, 16_000_000, 16), (20, 1_000_000, 16), (60, 1000, 16)):
        assert L.tenex_te_workspace_bytes(n, T, b) < L.tenex_te_pairs_workspace_bytes(n, T, b) + 256
    for n, T, b in ((20, 1_000_000, 6), (300, 2000, 6), (2000, 5000, 16), (10_000, 20_000, 38)):
        assert L.tenex_te_workspace_bytes(n, T, b) > L.tenex_te_pairs_workspace_bytes(n, T, b) + n * T // 8


def test_finite_check_in_a_forked_process(monkeypatch):
    """Arrays of a million elements are checked on host threads, which a forked child of a
    process that has them does not have."""
    monkeypatch.setattr(D, "_copy_workers", 8)
    monkeypatch.setattr(D, "_copy_pool", None)
    a = np.zeros(3 << 19)
    assert D.all_finite(a)
    ready = threading.Barrier(9)
    tasks = [D._pool().submit(ready.wait, 20) for _ in range(8)]
    ready.wait(20)
    assert len([t.result() for t in tasks]) == 8          # all threads are up
    assert D.all_finite(a)
    pid = os.fork()
    if pid == 0:
        threading.Timer(20, os._exit, (3,)).start()
        os._exit(0 if D.all_finite(a) and not D.all_finite(np.append(a, np.nan)) else 2)
    assert os.waitstatus_to_exitcode(os.waitpid(pid, 0)[1]) == 0


def test_permutations_are_sorted_one_by_one_when_memory_is_short(monkeypatch):
    from tenex_b200.inference.surrogate_test import build_block_perm
    want = build_block_perm(6, 400, "block", 10, 2, 9, 5, "cpu")[0]
    real = torch.argsort

    def argsort(x, **kw):
        if x.shape[0] > 6:
            raise torch.OutOfMemoryError("no room")
        return real(x, **kw)

    monkeypatch.setattr(torch, "argsort", argsort)
    assert torch.equal(build_block_perm(6, 400, "block", 10, 2, 9, 5, "cpu")[0], want)
    monkeypatch.setattr(torch, "argsort", lambda *a, **k: (_ for _ in ()).throw(
        torch.OutOfMemoryError("no room")))
    with pytest.raises(torch.OutOfMemoryError):
        build_block_perm(6, 400, "block", 10, 2, 9, 5, "cpu")


@pytest.mark.parametrize("size", [1, (5 << 19) - 1, 5 << 19, (5 << 19) + 1, (1 << 22) + 3])
def test_finite_check_around_the_size_where_threads_take_part(monkeypatch, size):
    used = []
    pool = D._pool()
    monkeypatch.setattr(D, "_pool", lambda: (used.append(1), pool)[1])
    a = np.zeros(size, np.float32)
    assert D.all_finite(a) and bool(used) == (size >= 5 << 19)
    for at in (0, size // 2, size - 1):
        for bad in (np.nan, np.inf, -np.inf):
            a[at] = bad
            assert not D.all_finite(a)
        a[at] = 0


def test_finite_check_of_a_large_array_in_a_forked_process():
    a = np.zeros(1 << 22, np.float32)
    assert D.all_finite(a)
    ready = threading.Barrier(D._copy_workers + 1)
    tasks = [D._pool().submit(ready.wait, 20) for _ in range(D._copy_workers)]
    ready.wait(20)
    assert len([t.result() for t in tasks]) == D._copy_workers and D.all_finite(a)
    pid = os.fork()
    if pid == 0:
        threading.Timer(20, os._exit, (3,)).start()
        os._exit(0 if D.all_finite(a) else 2)
    assert os.waitstatus_to_exitcode(os.waitpid(pid, 0)[1]) == 0


def test_workspace_has_the_tables_where_a_few_genes_have_many_bins():
    """A bin limit above 16 mostly comes from a few genes: the tensor-core path is worth it for
    smaller problems than at a limit of 16."""
    L = native.lib()
    for n, T in ((283, 5516), (311, 3714), (230, 1775)):
        least = L.tenex_te_pairs_workspace_bytes(n, T, 38)
        assert L.tenex_te_workspace_bytes(n, T, 38) > least + n * T // 8
        least = L.tenex_te_pairs_workspace_bytes(n, T, 16)
        assert L.tenex_te_workspace_bytes(n, T, 16) < least + 256

"""Threads that run plans and solves of different sizes at once: launches take
different amounts of shared memory, and each thread gets what a single one
gets, bit for bit."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_sizes_mixed_over_threads():
    from netsci_gb300 import device

    def solve(n):
        A = torch.full((n, n), float("inf"))
        i = torch.arange(n)
        for hop in (1, 7):
            A[i, (i + hop) % n] = A[(i + hop) % n, i] = 1.0 + (i % 5).float()
        A.fill_diagonal_(0)
        return device.apsp_lengths(A.cuda(), 12)[0]

    def score(m):
        X, _ = device.pack_trajectory(np.random.default_rng(m).standard_normal((6, 3 * m)), 3)
        ab = [(a, b) for a in range(6) for b in range(a, 6)]
        mi = torch.empty(len(ab), device="cuda")
        device.ksg_pairs(device.make_pairs(X, m, ab), 4, 3, mi=mi)
        return mi

    work = [(solve, n) for n in (64, 900, 2000, 3300)] + [(score, m) for m in (150, 700, 1500, 5000)]
    want = [f(size).cpu() for f, size in work]
    got = [[None] * 8 for _ in work]

    def run(w):
        f, size = work[w]
        with torch.cuda.stream(torch.cuda.Stream()):
            for r in range(8):
                got[w][r] = f(size)
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=run, args=(w,)) for w in range(len(work))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for w in range(len(work)):
        for r in range(8):
            assert got[w][r] is not None and torch.equal(got[w][r].cpu(), want[w])

"""GPU test of cpsd_overlap_tn's pooled workspaces: calls of several sizes on
several threads and streams at once give what they give alone, call after call.

Tolerance: exact (each call's sums have a fixed order)."""
import threading

import pytest

from cpsd_b200 import api

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_concurrent_calls_equal_single_ones():
    g = torch.Generator(device="cuda").manual_seed(3)
    sizes = [(128, 128, 4992), (37, 100, 3001), (3, 5, 130), (256, 64, 20000)]
    data = [(torch.randn(m, k, dtype=torch.float64, device="cuda", generator=g),
             torch.randn(n, k, dtype=torch.float64, device="cuda", generator=g)) for m, n, k in sizes]
    alone = [api.overlap_tn(a, b).clone() for a, b in data]
    for (a, b), c in zip(data, alone):
        assert (c - a @ b.T).abs().max().item() < 1e-12 * a.shape[1]
    bad = []

    def work(i):
        s = torch.cuda.Stream()
        for _ in range(20):
            if not torch.equal(api.overlap_tn(*data[i], stream=s.cuda_stream), alone[i]):
                bad.append(i)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad

"""Gradients of long virtual ranges in several threads, each with a context of its own:
the shared memory of a launch does not depend on what another thread launches."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_gradients_of_long_virtual_ranges():
    import torch

    import corr_gb300

    results = {}

    def work(v):
        try:
            r = np.random.default_rng(v)
            B = torch.from_numpy(0.1 * r.standard_normal((3, 1, v))).cuda()
            eps = torch.from_numpy(np.concatenate([[-1.0], r.uniform(0.1, 3.0, v)])).cuda()
            with corr_gb300.Context(0) as c:
                results[v] = [c.rimp2_gradient(B, eps, 1, v, 3)[0] for _ in range(250)]
        except Exception as e:  # reported by the main thread
            results[v] = e

    sizes = (4200, 5200, 5700, 6144)
    threads = [threading.Thread(target=work, args=(v,)) for v in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for v in sizes:
        assert isinstance(results[v], list), (v, results[v])
        assert np.ptp(results[v]) <= 1e-13 * abs(results[v][0])

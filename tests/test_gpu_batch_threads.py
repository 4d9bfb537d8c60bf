"""Batches of very different size run from two threads at once, each with its
own context: a large and a small batch use the same kernel with other amounts
of shared memory, and neither may disturb the other's launch."""
import threading

import numpy as np
import pytest

from energy_level_b200 import configs

pytestmark = pytest.mark.gpu


def _instance(n, seed):
    rng = np.random.default_rng(seed)
    calib = configs.calib_from_positions(configs.chain_positions(n, a=5.5, jitter=rng.uniform(-0.2, 0.2, n)))
    return dict(calib=calib, Om=np.full(n, 2.0), delta=-rng.uniform(0.0, 4.0, n), edges=configs.chain_edges(n))


@pytest.mark.parametrize("coop", [False, True])
def test_large_and_small_batch_in_two_threads(coop):
    from energy_level_b200.batched import BatchedGroundStates
    # the same instantiation on both sides: one CTA of 512 threads per SM
    # (FP32, 28,657 rows = 112 KB next to 144 rows), or 64 rows per CTA
    # (FP64, Krylov slices of 160 and of 8 vectors)
    sizes = {"large": (21, 4), "small": (10, 4)} if not coop else {"large": (16, 160), "small": (16, 8)}
    loops = 400 if coop else 4000
    out, errors = {}, []
    start, done = threading.Barrier(2), threading.Event()

    def work(name):
        n, m = sizes[name]
        try:
            b = BatchedGroundStates([_instance(n, 3)], dtype="float64" if coop else "float32", max_iter=m)
            go = (lambda: b.run_coop(seed=1)) if coop else (lambda: b.run(threads=512, ctas_per_sm=1, seed=1))
            go()
            first = b.results()["E0"].copy()
            start.wait(60)
            for _ in range(loops if name == "large" else 100 * loops):
                go()
                if name == "small" and done.is_set():
                    break
            done.set()
            out[name] = (first, b.results()["E0"].copy())
            b.close()
        except Exception as e:      # noqa: BLE001 - reported below
            errors.append((name, repr(e)))
            start.abort()
            done.set()

    threads = [threading.Thread(target=work, args=(name,)) for name in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for first, last in out.values():
        assert np.array_equal(first, last)

"""Two host threads on their own streams, one with hexa-double and one with
double- or quad-double problems, over every route whose kernels take shared
memory by the number of digits: sum planes (whole diagonals and prefix sums),
digit pairs, batches, the plain batch."""
import threading

import pytest

from conftest import pkg


@pytest.mark.gpu
def test_two_threads_of_different_limb_counts():
    import torch
    api = pkg("api")

    def work(p, shapes):
        ops = [(api.generate("uniform", p, m, k, 51), api.generate("normal", p, k, n, 52))
               for m, n, k in shapes]
        small = [(a[:40, :50].contiguous(), b[:50, :30].contiguous()) for a, b in ops]
        plan = api.BatchPlan(small)

        def run(stream):
            out = [api.gemm(a, b, stream=stream) for a, b in ops]
            out += [c.clone() for c in plan.run(stream=stream)]
            out += api.gemm_batched(small, "plain", stream=stream)
            return out

        return run

    runs = [work(16, [(768, 512, 512), (100, 90, 80)]),
            work(4, [(768, 800, 1024), (100, 90, 80)]), ]
    torch.cuda.synchronize()
    main = torch.cuda.current_stream()
    want = [run(main) for run in runs]
    torch.cuda.synchronize()
    errors = []

    def worker(t):
        stream = torch.cuda.Stream()
        try:
            with torch.cuda.stream(stream):
                for _ in range(30):
                    got = runs[t](stream)
                    stream.synchronize()
                    if not all(torch.equal(a, b) for a, b in zip(got, want[t])):
                        raise AssertionError("other bits")
                    stream.synchronize()
        except Exception as e:  # reported on the main thread
            errors.append((t, e))

    threads = [threading.Thread(target=worker, args=(t,)) for t in range(2)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors, errors
    assert api.device_status() == 0

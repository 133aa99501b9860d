"""A captured mdg_batch_run replayed after the plan's units were dealt anew: under
the other split mode and under the other single-CTA tile policies the graph's
launch takes the present units."""
import pytest

from conftest import pkg


@pytest.mark.gpu
@pytest.mark.parametrize("first", ["256", "pair"])
def test_replay_after_the_units_changed(first):
    import torch
    api = pkg("api")
    ops = [(api.generate("uniform", p, m, k, i), api.generate("normal", p, k, n, i + 9))
           for i, (p, m, n, k) in enumerate([(2, 40, 40, 40), (8, 300, 200, 130), (4, 70, 300, 65)])]
    plan = api.BatchPlan(ops)
    plan.set_tiles(first)
    want = [c.clone() for c in plan.run()]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.run()
    changes = [lambda: plan.set_split(False), lambda: plan.set_split(True)]
    if first != "pair":
        changes += [lambda: plan.set_tiles("128"), lambda: plan.set_split(False),
                    lambda: plan.set_tiles("auto")]
    for change in changes:
        change()
        for c in plan.Cs:
            c.fill_(-1.0)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(plan.Cs, want))
    assert api.device_status() == 0

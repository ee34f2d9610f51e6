"""A per-angle plan that is captured into a caller's graph keeps its launches in that graph:
other per-angle plans of the scene execute on streams of their own meanwhile, and the graph
computes the same fields."""
import numpy as np
import pytest

import sagittasbr_b200 as sbr
from sagittasbr_b200 import meshes as M
from sagittasbr_b200.sharding import _DeviceArray

pytestmark = pytest.mark.gpu


def test_other_plans_run_while_one_is_captured():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    v, t = M.plate_cluster(6, 4, seed=9)
    n = 20
    th, ph = np.full(n, 70.0), np.linspace(0.0, 330.0, n)
    jobs = [sbr.JobSpec(th, ph, [1e9, 2e9], 64, 57, 2.2, 4), sbr.JobSpec(th, ph + 5.0, [1e9, 2e9], 64, 57, 2.2, 4)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    with sbr.Scene(v, t) as s:
        want = [sbr.run(s, j, mode=sbr.MODE_PER_ANGLE) for j in jobs]
        plans = [sbr.Plan(s, [j], mode=sbr.MODE_PER_ANGLE, stream=q.cuda_stream) for j, q in zip(jobs, streams)]
        for p in plans:
            p.execute()
            p.results()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=streams[0], capture_error_mode="thread_local"):
            plans[0].execute()
            plans[1].execute()
        np.testing.assert_array_equal(plans[1].results().field, want[1].field)
        field = torch.as_tensor(_DeviceArray(plans[0].device_results()[0], 4 * n), device="cuda")
        for _ in range(2):
            field.zero_()
            graph.replay()
            torch.cuda.synchronize()
            f = field.cpu().numpy()
            np.testing.assert_array_equal(f[0::2] + 1j * f[1::2], want[0].field)
        del graph
        for p in plans:
            p.close()

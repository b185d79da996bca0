"""A job list used right after it was set, on a stream that does not wait for
the legacy one, and by calls that are captured."""
import numpy as np
import pytest
import torch

from nr_gpu_ldpc_gb300.batch import Batch, make_jobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 26, 700])  # clusters; the persistent kernel
def test_list_set_then_used_on_side_streams_and_in_graphs(gpu, n):
    b = Batch(max_jobs=n)
    llr_e = torch.empty(66 * 384 * n, device=gpu).normal_(generator=torch.Generator(device=gpu).manual_seed(n)) * 2 + 2
    side, got = torch.cuda.Stream(), {}
    for way in ("legacy", "side", "graph"):
        for z in (384, 64):  # the second list replaces one that ran
            jobs, n_llr, _, n_out = make_jobs(np.full(n, 1), z)
            llr, out = torch.empty(n_llr, device=gpu), torch.zeros(n_out, dtype=torch.uint8, device=gpu)
            torch.cuda.synchronize()
            b.set_jobs(jobs)
            if way == "graph":
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph):
                    b.derate(llr_e, llr)
                    b.decode(llr, out, 5)
                graph.replay()
            else:
                stream = side if way == "side" else torch.cuda.default_stream()
                b.derate(llr_e, llr, stream=stream)
                b.decode(llr, out, 5, stream=stream)
            torch.cuda.synchronize()
            assert torch.equal(out, got.setdefault(z, out)) and b.device_error() == 0
    b.close()

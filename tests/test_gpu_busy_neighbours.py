"""Small batches choose their kernel by what other decoders have in flight on
other streams: the bits are those of a call alone, also while one of the
streams is captured."""
import numpy as np
import pytest
import torch

from nr_gpu_ldpc_gb300 import Decoder, codes
from nr_gpu_ldpc_gb300.batch import Batch, make_jobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 20, 40])
def test_small_batches_on_several_streams(gpu, n):
    sig = torch.full((n,), codes.noise_sigma(1.8, 1 / 3), device=gpu)
    decs = [Decoder(bg=1, z=384, max_batch=n) for _ in range(4)]
    jobs, n_llr, _, n_out = make_jobs(np.full(n, 2), 208)
    lists = [Batch(max_jobs=n) for _ in range(2)]
    for b in lists:
        b.set_jobs(jobs)
    llr = [decs[0].gen_llr(seed=k, cw_base=0, sigma=sig)[0] for k in range(4)]
    mother = torch.randn(n_llr, device=gpu) + 1.0
    want = []
    for d, x in zip(decs, llr):
        want.append(d.decode(x, 10).clone())
        torch.cuda.synchronize()
    out_b = [torch.zeros(n_out, dtype=torch.uint8, device=gpu) for _ in lists]
    lists[0].decode(mother, out_b[0], 10)
    torch.cuda.synchronize()
    want_b = out_b[0].clone()
    streams = [torch.cuda.Stream() for _ in range(6)]
    for _ in range(5):
        got = []
        for d, x, s in zip(decs, llr, streams):
            with torch.cuda.stream(s):
                got.append(d.decode(x, 10))
        for b, o, s in zip(lists, out_b, streams[4:]):
            with torch.cuda.stream(s):
                o.zero_()
                b.decode(mother, o, 10)
        torch.cuda.synchronize()
        assert all(torch.equal(g, w) for g, w in zip(got, want))
        assert all(torch.equal(o, want_b) for o in out_b)
    # neighbours busy while a call is captured, then the captured call replayed
    graph, out = torch.cuda.CUDAGraph(), torch.zeros_like(want[0])
    with torch.cuda.stream(streams[1]):
        keep = [decs[1].decode(llr[1], 10) for _ in range(3)]
    with torch.cuda.graph(graph):
        out.copy_(decs[0].decode(llr[0], 10))
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want[0]) and all(torch.equal(k, want[1]) for k in keep)

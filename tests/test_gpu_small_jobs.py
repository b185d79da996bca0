"""Short job lists (one codeword on a cluster of CTAs), de-rate-matching at the
edges of the circular buffer and CRCs at the edges of a warp's stretches."""
import ctypes as C

import numpy as np
import pytest
import torch

from nr_gpu_ldpc_gb300 import _lib, codes
from nr_gpu_ldpc_gb300.batch import Batch, make_jobs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _decode(batch, jobs, llr, n_out, n, it):
    packed = torch.zeros(n_out, dtype=torch.uint8, device="cuda")
    iters = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    batch.set_jobs(jobs)
    batch.decode(llr, packed, it, early_stop=True, iters=iters)
    torch.cuda.synchronize()
    return packed.cpu().numpy(), iters.cpu().numpy()


def test_short_lists_equal_the_long_list():
    # 1,000 jobs run in the persistent kernel; pieces of the list on clusters,
    # of several sizes and in several rounds
    rng = np.random.default_rng(8)
    n = 1000
    bg, z = rng.integers(1, 3, n), rng.choice([2, 7, 13, 40, 64, 208, 384], n)
    jobs, n_llr, _, n_out = make_jobs(bg, z)
    llr = torch.empty(n_llr, device="cuda").normal_(generator=torch.Generator(device="cuda").manual_seed(2)) * 2 + 2
    b = Batch(max_jobs=n)
    want, want_it = _decode(b, jobs, llr, n_out, n, 7)
    for lo, k in ((0, 1), (1, 3), (4, 8), (12, 26), (40, 47), (90, 80), (200, 160), (400, 300)):
        got, it = _decode(b, jobs[lo:lo + k], llr, n_out, k, 7)
        assert np.array_equal(it, want_it[lo:lo + k]), (lo, k)
        for j in jobs[lo:lo + k]:
            o = int(j["out_offset"])
            e = o + (codes.BG_SHAPE[int(j["bg"])][1] * int(j["z"]) + 7) // 8
            assert np.array_equal(got[o:e], want[o:e]), (lo, k)
        # nothing outside the pieces' own bytes is written
        first, last = int(jobs[lo]["out_offset"]), int(jobs[lo + k]["out_offset"])
        assert not got[:first].any() and not got[last:].any()


@pytest.mark.parametrize("bg,z,fill", [(1, 384, 24), (2, 384, 0), (2, 7, 3), (1, 64, 39)])
@pytest.mark.parametrize("qm", [1, 6])
def test_derate_at_the_buffer_edges(bg, z, fill, qm):
    kb = codes.KB_MAX[bg]
    kp = kb * z - fill
    nc = (66 if bg == 1 else 50) * z - fill
    es = sorted({max(qm, e // qm * qm) for e in (qm, nc - qm, nc, nc + qm, 2 * nc, 3 * nc + qm, kp // 2)})
    oc = O.OracleCode(codes.base_matrix(bg, codes.set_index(z)), z)
    rng = np.random.default_rng(z)
    for rv in (0, 3):
        jobs, n_llr, n_e, _ = make_jobs(np.full(len(es), bg), z, k_prime=kp, e=np.array(es), rv=rv, qm=qm)
        x = rng.normal(0, 3, n_e).astype(np.float32)
        b = Batch(max_jobs=len(es))
        b.set_jobs(jobs)
        llr = torch.full((n_llr,), 7.0, device="cuda")
        b.derate(torch.from_numpy(x).cuda(), llr)
        h = llr.cpu().numpy()
        for j in jobs:
            e, at = int(j["e"]), int(j["e_offset"])
            want = O.derate_match(oc, kb, bg, x[None, at:at + e], kp, e, rv, qm)[0]
            got = h[j["llr_offset"]:j["llr_offset"] + oc.n_bp]
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (rv, e)


@pytest.mark.parametrize("n_bits", [1, 7, 9, 255, 256, 257, 264, 2047, 2056, 8424, 8429])
def test_crc_at_the_stretch_edges(n_bits):
    rng = np.random.default_rng(n_bits)
    stride = (n_bits + 7) // 8 + 1
    for n in (1, 8, 9):
        data = rng.integers(0, 256, (n, stride), dtype=np.uint8)
        d = torch.from_numpy(data).cuda()
        rem = torch.empty(n, dtype=torch.int32, device="cuda")
        for ctype, poly in enumerate((O.CRC24A, O.CRC24B, O.CRC16)):
            assert _lib.load().nrldpc_crc(C.c_void_p(d.data_ptr()), n, stride, n_bits, ctype,
                                          C.c_void_p(rem.data_ptr()),
                                          C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
            want = np.array([O.crc(r, n_bits, poly) for r in data], np.uint32)
            assert np.array_equal(rem.cpu().numpy().astype(np.uint32), want)

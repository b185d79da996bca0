"""The small-batch decoder's waits for counted bytes are bounded.  The self-test
tells the first CTA of every cluster to expect 16 bytes more than are sent: its
wait runs out, then those of the CTAs that wait for it; the error is reported,
nothing is written, and the handle decodes bit-exactly afterwards."""
import ctypes as C

import numpy as np
import pytest
import torch

from nr_gpu_ldpc_gb300 import Decoder, _lib, codes
from nr_gpu_ldpc_gb300.batch import Batch, make_jobs
from oracle.oracle import OracleCode

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bg,z,n", [(1, 384, 1), (1, 384, 20), (2, 208, 9)])  # 20: more than are resident at once
def test_wait_that_runs_out_is_reported(gpu, bg, z, n):
    oc = OracleCode(codes.base_matrix(bg, codes.set_index(z)), z)
    kb, rate = (22, 1 / 3) if bg == 1 else (10, 1 / 5)
    llr, _ = oc.gen_llr(kb, 77, 0, np.full(n, codes.noise_sigma(2.0, rate), np.float32), 2)
    dec = Decoder(bg=bg, z=z, max_batch=n)
    d_llr = torch.from_numpy(llr).to(gpu)
    for _ in range(2):
        out = torch.full((n, dec.packed_bytes), 0xA5, dtype=torch.uint8, device=gpu)
        assert _lib.load().nrldpc_selftest_split_timeout(
            dec._h, C.c_void_p(d_llr.data_ptr()), C.c_void_p(out.data_ptr()), n,
            C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        torch.cuda.synchronize()
        assert dec.device_error() == -6 and dec.device_error() == 0  # NRLDPC_ERR_TIMEOUT, cleared by the read
        assert torch.all(out == 0xA5)
        packed = dec.decode(d_llr, 5)
        torch.cuda.synchronize()
        assert np.array_equal(packed.cpu().numpy(), oc.minsum_f32(llr, 5)[0])
        assert dec.device_error() == 0
    dec.close()


def test_code_without_such_clusters(gpu):
    # 12 rows of 24 sub-rows: one CTA holds the code, nothing is sent
    dec = Decoder(base=codes.wifi_base(), z=24, max_batch=1)
    llr = torch.zeros(dec.n_bp, device=gpu)
    out = torch.zeros(dec.packed_bytes, dtype=torch.uint8, device=gpu)
    assert _lib.load().nrldpc_selftest_split_timeout(dec._h, C.c_void_p(llr.data_ptr()), C.c_void_p(out.data_ptr()),
                                                     1, None) == -2  # NRLDPC_ERR_BAD_CONFIG
    dec.close()


@pytest.mark.parametrize("bg,z,n", [(1, 384, 1), (1, 384, 12), (2, 208, 9)])
def test_wait_that_runs_out_in_a_job_list(gpu, bg, z, n):
    jobs, n_llr, _, n_out = make_jobs(np.full(n, bg), z)
    llr = torch.empty(n_llr, device=gpu).normal_(generator=torch.Generator(device=gpu).manual_seed(3)) * 2 + 2
    b = Batch(max_jobs=n)
    b.set_jobs(jobs)
    want, out = (torch.full((n_out,), 0xA5, dtype=torch.uint8, device=gpu) for _ in range(2))
    b.decode(llr, want, 5)
    assert b.device_error() == 0
    assert _lib.load().nrldpc_selftest_batch_timeout(b._h, C.c_void_p(llr.data_ptr()), C.c_void_p(out.data_ptr()),
                                                     C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    assert b.device_error() == -6 and b.device_error() == 0
    assert torch.all(out == 0xA5)
    b.decode(llr, out, 5)
    assert torch.equal(out, want) and b.device_error() == 0
    b.close()

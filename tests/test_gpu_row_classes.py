"""decode_kernel is compiled for codes whose rows are like BG1's or BG2's
(degrees, and which of them end in a suffix column) and for any other: every
class, at sizes around its geometry (cw_per_cta, ragged warps), against the
oracle bit for bit."""
import numpy as np
import pytest
import torch

from nr_gpu_ldpc_gb300 import Decoder, codes
from nr_gpu_ldpc_gb300.batch import Batch, make_jobs
from oracle.oracle import OracleCode

pytestmark = pytest.mark.gpu


def _base(bg, z, change):
    base = np.array(codes.base_matrix(bg, codes.set_index(z)), dtype=np.int32)
    deg = (base >= 0).sum(1)
    if change == "degree":  # a row of a degree that the class does not have
        r = int(np.flatnonzero(deg == (10 if bg == 1 else 6))[-1])
        base[r, int(np.flatnonzero(base[r, :10] < 0)[0])] = 5
    elif change == "suffix":  # the last column is no suffix any more: its row ends in a core column
        r = int(np.flatnonzero(deg == 3)[0])
        base[r, -1] = 7
    elif change == "swap":  # a row of a suffix degree without a suffix column
        r = 4 if bg == 1 else 5
        c = int(np.flatnonzero(base[r] >= 0)[-1])
        base[r - 1, c] = 3  # column of degree 2
    return base


@pytest.mark.parametrize("bg,z,change,n", [
    (1, 384, None, 310), (1, 208, None, 460), (1, 56, None, 700), (1, 7, None, 700),
    (2, 384, None, 310), (2, 208, None, 460), (2, 56, None, 700), (2, 7, None, 700),
    (1, 56, "degree", 700), (2, 56, "degree", 700), (1, 24, "suffix", 700), (2, 24, "suffix", 700),
    (2, 24, "swap", 700),
])
def test_row_classes_against_oracle(gpu, bg, z, change, n):
    base = _base(bg, z, change)
    rng = np.random.default_rng(bg * 1000 + z)
    for cpb in (0, 1):
        dec = Decoder(base=base, z=z, max_batch=n, cw_per_cta=cpb)
        oc = OracleCode(base, z)
        # a noisy all-zero codeword: some rows converge, some do not
        llr = (1.1 + rng.standard_normal((n, dec.n_bp)) * rng.uniform(0.4, 1.4, (n, 1))).astype(np.float32)
        llr[:, : 2 * z] = 0.0
        d_llr = torch.from_numpy(llr).to(gpu)
        pk, app, it = dec.decode(d_llr, 4, early_stop=True, want_app=True, want_iters=True)
        dec.set_schedule("layered")
        pl = dec.decode(d_llr, 2)
        torch.cuda.synchronize()
        opk, oapp, oit = oc.minsum_f32(llr, 4, early_stop=True, want_app=True, threads=8)
        np.testing.assert_array_equal(pk.cpu().numpy(), opk)
        np.testing.assert_array_equal(app.cpu().numpy(), oapp)
        np.testing.assert_array_equal(it.cpu().numpy(), oit)
        opl, _, _ = oc.layered_f32(llr, 2, threads=8)
        np.testing.assert_array_equal(pl.cpu().numpy(), opl)
        dec.close()


@pytest.mark.parametrize("spt", [1, 2])
def test_job_list_of_both_classes_equals_single_code_decodes(gpu, spt):
    """spt 2 for one code of the list: the whole list takes the kernel for any
    code."""
    shapes = [(bg, z) for bg in (1, 2) for z in (2, 7, 56, 208, 384)]
    per = 160
    bg = np.repeat([s[0] for s in shapes], per)
    z = np.repeat([s[1] for s in shapes], per)
    jobs, n_llr, _, n_out = make_jobs(bg, z)
    b = Batch(max_jobs=bg.size)
    b.set_sub_rows_per_thread(2, 56, spt)
    b.set_jobs(jobs)
    llr = torch.randn(n_llr, generator=torch.Generator().manual_seed(3)).to(gpu) + 0.9
    packed = torch.zeros(n_out, dtype=torch.uint8, device=gpu)
    iters = torch.zeros(bg.size, dtype=torch.int32, device=gpu)
    b.decode(llr, packed, 6, early_stop=True, iters=iters)
    torch.cuda.synchronize()
    for k, (g, size) in enumerate(shapes):
        dec = Decoder(bg=g, z=size, max_batch=per)
        at = jobs["llr_offset"][k * per: (k + 1) * per]
        own = torch.stack([llr[o: o + dec.n_bp] for o in at.tolist()]).contiguous()
        pk, it = dec.decode(own, 6, early_stop=True, want_iters=True)
        torch.cuda.synchronize()
        at = jobs["out_offset"][k * per: (k + 1) * per]
        got = torch.stack([packed[o: o + dec.packed_bytes] for o in at.tolist()])
        assert torch.equal(got, pk), (g, size)
        assert torch.equal(iters[k * per: (k + 1) * per], it), (g, size)
        dec.close()
    b.close()

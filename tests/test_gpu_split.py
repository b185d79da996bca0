"""Small batches (one codeword on a cluster of CTAs) against the oracle and
against the same codewords inside a batch that fills the GPU: hard decisions,
posteriors and iteration counts, bit for bit.  Batch sizes lie at the edges of
the cluster sizes (16, 10, 8, 6, 5, 4, 3, 2, 1 CTAs per codeword, several
rounds), lifting sizes on both sides of a warp's 32 sub-rows and at codes
whose rows run in phases."""
import numpy as np
import pytest
import torch

from nr_gpu_ldpc_gb300 import Decoder, codes
from oracle.oracle import OracleCode

pytestmark = pytest.mark.gpu


def _llrs(oc, bg, n, seed, ebn0=2.0):
    kb, rate = (22, 1 / 3) if bg == 1 else (10, 1 / 5)
    return oc.gen_llr(kb, seed, 0, np.full(n, codes.noise_sigma(ebn0, rate), np.float32), 2)[0]


def _bits(a):
    """fp32 bit patterns, every NaN as one (its payload is unspecified)."""
    b = np.ascontiguousarray(a, np.float32).view(np.uint32).copy()
    b[np.isnan(a)] = 0x7FC00000
    return b


def _check(dec, oc, llr, it, es, ref=None, weights=None):
    want = ref or (oc.wms_decode_f32(llr, it, weights, early_stop=es, want_app=True) if weights is not None else
                   oc.minsum_f32(llr, it, early_stop=es, want_app=True, threads=16))
    pk, app, its = dec.decode(torch.from_numpy(llr).cuda(), it, early_stop=es, want_app=True, want_iters=True,
                              weighted=weights is not None)
    assert np.array_equal(pk.cpu().numpy(), want[0])
    assert np.array_equal(_bits(app.cpu().numpy()), _bits(want[1]))
    assert np.array_equal(its.cpu().numpy(), want[2])
    assert dec.device_error() == 0


@pytest.mark.parametrize("bg,z", [(1, 384), (2, 384), (1, 352), (1, 208), (2, 36), (1, 72), (2, 13), (1, 2)])
@pytest.mark.parametrize("es", [False, True])
def test_batch_sizes_at_the_cluster_edges(bg, z, es):
    oc = OracleCode(codes.base_matrix(bg, codes.set_index(z)), z)
    llr = _llrs(oc, bg, 80, 5)
    ref = oc.minsum_f32(llr, 6, early_stop=es, want_app=True, threads=16)
    dec = Decoder(bg=bg, z=z, max_batch=80)
    for n in (1, 7, 8, 13, 16, 24, 28, 29, 36, 37, 46, 47, 77, 80):
        _check(dec, oc, llr[:n], 6, es, ref=tuple(r[:n] for r in ref))
    dec.close()


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("bg,z,n", [(1, 384, 620), (2, 40, 3000), (1, 96, 1300)])
def test_same_bits_as_in_a_full_batch(bg, z, n, weighted):
    dec = Decoder(bg=bg, z=z, max_batch=n)
    if weighted:
        dec.set_weights(np.random.default_rng(z).uniform(0.6, 0.95, (5, dec.n_edges)))
    sig = torch.full((n,), codes.noise_sigma(1.9, 1 / 3 if bg == 1 else 1 / 5), device="cuda")
    llr, _ = dec.gen_llr(seed=9, cw_base=0, sigma=sig)
    big = dec.decode(llr, 8, early_stop=True, want_app=True, want_iters=True, weighted=weighted)
    for lo, k in ((0, 1), (3, 5), (40, 12), (100, 30), (200, 44), (300, 150)):
        small = dec.decode(llr[lo:lo + k], 8, early_stop=True, want_app=True, want_iters=True, weighted=weighted)
        for a, b in zip(small, big):
            assert torch.equal(a, b[lo:lo + k])
    dec.close()


@pytest.mark.parametrize("n", [1, 9, 40])
def test_special_values_custom_code_and_weights(n):
    # a matrix whose last columns are not all suffixes, and values the minima
    # and signs treat specially: +-0, infinities, NaN, beyond the 1000 start
    rng = np.random.default_rng(n)
    for base, z, dec in ((codes.wifi_base(), 96, Decoder(base=codes.wifi_base(), z=96, max_batch=n)),
                         (codes.base_matrix(1, codes.set_index(384)), 384, Decoder(bg=1, z=384, max_batch=n))):
        oc = OracleCode(base, z)
        llr = rng.normal(0, 4, (n, oc.n_bp)).astype(np.float32)
        for v in (0.0, -0.0, np.inf, -np.inf, np.nan, 1500.0, -1000.0):
            llr[rng.random(llr.shape) < 0.02] = v
        _check(dec, oc, llr, 3, False)
        w = rng.uniform(-0.2, 1.0, (2, oc.n_edges)).astype(np.float32)
        dec.set_weights(w)
        _check(dec, oc, llr, 4, True, weights=w)
        dec.close()


@pytest.mark.parametrize("n", [1, 12, 40])
def test_host_buffers(n):
    z = 384
    oc = OracleCode(codes.base_matrix(1, codes.set_index(z)), z)
    llr = _llrs(oc, 1, n, 3)
    want = oc.minsum_f32(llr, 5, threads=16)[0]
    dec = Decoder(bg=1, z=z, max_batch=n)
    host = torch.from_numpy(llr).pin_memory()
    for mode in ("auto", "copy", "direct"):
        out = torch.zeros((n, oc.n_bytes), dtype=torch.uint8).pin_memory()
        dec.set_host_transfer(mode)
        dec.decode_host(host, out, 5)
        torch.cuda.synchronize()
        assert np.array_equal(out.numpy(), want), mode
    dec.close()


def test_captured_in_a_graph():
    # the small-batch path allocates nothing and may be captured and replayed
    dec = Decoder(bg=2, z=128, max_batch=16)
    sig = torch.full((16,), codes.noise_sigma(2.0, 1 / 5), device="cuda")
    llr, _ = dec.gen_llr(seed=4, cw_base=0, sigma=sig)
    want = dec.decode(llr, 5)
    out = torch.zeros_like(want)
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        dec.decode(llr, 5, out=out)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    dec.close()

"""Training loss and weight gradients at the edges of the kernels' shapes: rows
of 19 edges (in a loop) and of up to 10 (unrolled), codeword groups that are not
full, threads without a codeword (Z not a multiple of 32)."""
import numpy as np
import pytest
import torch

from nr_gpu_ldpc_gb300 import Trainer, codes
from oracle.oracle import OracleCode

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bg,z,n", [(1, 384, 3), (1, 36, 11), (2, 13, 31), (2, 384, 2), (1, 2, 5)])
@pytest.mark.parametrize("schedule", ["flooding", "layered"])
def test_loss_and_gradient_match_oracle(bg, z, n, schedule):
    layered, T = schedule == "layered", 3
    oc = OracleCode(codes.base_matrix(bg, codes.set_index(z)), z)
    kb, rate = (22, 1 / 3) if bg == 1 else (10, 1 / 5)
    llr, cw = oc.gen_llr(kb, 17 + z, 0, np.full(n, codes.noise_sigma(1.5, rate), np.float32), 2)
    rng = np.random.default_rng(z)
    # no two |Q| tie exactly in place of the punctured zeros
    llr[:, :2 * z] = rng.normal(0, 0.3, (n, 2 * z)).astype(np.float32)
    w = rng.uniform(0.55, 0.95, (T, oc.n_edges)).astype(np.float32)
    tr = Trainer(bg=bg, z=z, n_iter=T, batch=n, chunk=n, schedule=schedule)
    loss, grad = tr.loss_and_grad(torch.from_numpy(llr).cuda(), torch.from_numpy(cw).cuda(), torch.from_numpy(w).cuda())
    want, want_grad, _ = oc.wms_loss_grad(llr, cw, T, w.astype(np.float64), layered=layered, f32_forward=layered)
    assert abs(loss - want) <= 1e-5 * abs(want)
    rel = np.linalg.norm(grad.cpu().numpy() - want_grad) / np.linalg.norm(want_grad)
    # flooding: against a 64-bit forward, whose argmins can differ in near ties
    assert rel < (2e-4 if layered else 2e-3), rel

"""The proposal network's convolutions over row tiles that a batch fills partly or several times.

A pair's outputs do not depend on its batch (each accumulator sums the same products in the same
order), so a batch's outputs equal the single pairs' bit for bit.  With a power of two of pairs the
loss gradient of each is its single gradient scaled exactly, also in BF16, so the batch's gradients are the
mean of the single ones up to the FP32 summation order: 1e-4 relative L2 for sums of up to 2^16 terms.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 8, 32])
def test_batch_equals_single_pairs(cuda, lib, n):
    import torch
    from cugridsearch_b200 import synthetic as S
    from cugridsearch_b200.proposal import ProposalNet
    f, m, _ = S.config4_batch(61, n, cuda, 128)
    labels = torch.from_numpy(np.random.default_rng(3).uniform(-1, 1, (n, 8)).astype(np.float32)).to(cuda)
    net = ProposalNet(max_batch=n, seed=5)
    out = net.forward(f, m).cpu().numpy().copy()
    net.backward(labels)
    grads = net.grads().astype(np.float64)
    mean = np.zeros_like(grads)
    for i in range(n):
        one = net.forward(f[i:i + 1].contiguous(), m[i:i + 1].contiguous()).cpu().numpy()
        np.testing.assert_array_equal(one[0], out[i])
        net.backward(labels[i:i + 1].contiguous())
        mean += net.grads().astype(np.float64) / n
    net.close()
    assert np.linalg.norm(grads - mean) <= 1e-4 * np.linalg.norm(mean)

"""The parameter sweep at the edges of its blocks (256 x 4 values) and over several waves of them."""
import pytest
import torch

from rembrandt_b200.ops import native_ops as K
from rembrandt_b200.optim.sgd import reference_step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 1023, 1024, 1025, 4 * 1184 * 1024 + 1, 9_700_003])
def test_every_value_is_updated_once_and_nothing_behind_them(n):
    torch.manual_seed(n)
    w, g, v = (torch.randn(n + 8, device="cuda") for _ in range(3))
    w16 = torch.full((n + 8,), 7.0, device="cuda", dtype=torch.bfloat16)
    before = [t[n:].clone() for t in (w, g, v, w16)]
    ref = reference_step(w[:n].clone(), g[:n].clone(), v[:n].clone(), lr=0.1, mu=0.9, l2=5e-4, grad_scale=0.5, mode=1)
    K.sgd_fused(w[:n], g[:n], v[:n], w16[:n], n, 0.1, 0.9, 5e-4, 0.5, 1)
    # four products and sums of values below 6 in 32 bits: 4 x 6 x 2^-23 < 3e-6, with the order of the operations open
    for got, want in zip((w, g, v), ref):
        assert (got[:n] - want).abs().max() < 1e-5
    assert torch.equal(w16[:n], w[:n].bfloat16())
    for t, kept in zip((w, g, v, w16), before):
        assert torch.equal(t[n:], kept)

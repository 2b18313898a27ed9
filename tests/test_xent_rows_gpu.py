"""The loss backward's two ways of moving rows (each thread its own, or a CTA's rows by way of shared
memory where scores and gradients are past what L2 keeps) give the same bits: a call past the line
against its two halves below it."""
import pytest
import torch

import armsparse_gb300 as A
from gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,classes,width", [(1 << 18, 64, 64), (1 << 18, 57, 64), (1 << 20, 47, 48),
                                             (1 << 20, 41, 48), (1 << 21, 30, 32)])
def test_halves_of_a_large_call(n, classes, width):
    gen = torch.Generator(device=dev()).manual_seed(n + classes)
    scores = torch.randn(n, width, generator=gen, device=dev()).bfloat16()
    labels = torch.randint(0, classes, (n,), generator=gen, device=dev())
    labels[::1001] = classes  # out of range: a zero gradient
    _, lse = A.softmax_xent(scores, labels, classes)
    with pytest.raises(A.NativeError):
        A.sync_status()
    whole = A.softmax_xent_grad(scores, labels, classes, lse, torch.ones((), device=dev()))
    h = n // 2
    half = torch.full((), 0.5, device=dev())  # gscale / n stays the same power of two
    parts = [A.softmax_xent_grad(scores[lo:lo + h], labels[lo:lo + h], classes, lse[lo:lo + h], half)
             for lo in (0, h)]
    assert torch.equal(whole.view(torch.int16), torch.cat(parts).view(torch.int16))
    assert not whole[:, classes:].any() and not whole[::1001].any()
    p = torch.softmax(scores[:999, :classes].float(), 1)
    p[torch.arange(999), labels[:999].clamp(max=classes - 1)] -= 1
    p[0] = 0  # the out-of-range label
    assert torch.allclose(whole[:999, :classes].float() * n, p, rtol=2 ** -7, atol=1e-6)
    A.sync_status()

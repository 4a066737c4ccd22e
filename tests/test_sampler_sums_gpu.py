"""Sampler kernel: what a row gives does not depend on the signs of zeros among the listed entries."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("cut", ["top_p", "top_k"])
def test_negative_zeros_below_a_maximum_of_eight(dtype, cut):
    """The list reaches to 8 below the maximum, here to 0: an entry of -0 is below that and cannot be kept in place of larger ones."""
    from tgi_b200.ops import cuda as K

    K.load()
    x = torch.full((64, 1000), -20.0, device="cuda")
    x[:, 100:300] = -0.0
    x[:, 7] = 8.0
    one = torch.ones(64, device="cuda")
    kw = {"top_p": {"top_p": one * 0.5}, "top_k": {"top_k": one.int()}}[cut]
    ids, lps = K.fused_sample(x.to(dtype), do_sample=one.to(torch.uint8), seeds=torch.arange(64, device="cuda"), steps=one.int(), **kw)
    assert (ids == 7).all() and (lps == 0).all()

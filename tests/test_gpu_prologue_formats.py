"""Forwards behind the fused prologues against the unfused sequence, bit for bit, where the library's choice of kernel and
code format depends on the shape: many tokens on packed weights (narrow and wide tiles), and 64 to 255 tokens on
prepared weights (where the tensor-core kernel can win on the prepared copy and lose on the packed arrays)."""

import pytest
import torch

from oracle import w4a4_oracle as O
from helpers import make_case
from zip_kernel_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,N,K,density,prepared", [
    (256, 640, 1024, 0.2, False), (300, 1000, 2048, 0.1, False), (257, 128 * 120, 384, 0.2, False), (513, 4096, 4096, 0.05, False),
    (128, 4864, 4096, 0.05, True), (64, 640, 512, 0.2, True), (255, 5120, 4096, 0.0, True), (257, 128 * 120, 384, 0.2, True)])
def test_prologue_forwards_equal_the_unfused_sequence(T, N, K, density, prepared):
    from zip_kernel_b200 import _lib, v9_linear
    dev = torch.device("cuda")
    W, X = make_case(T, N, K, density, perm_seed=3)
    Wd = W.to(dev)
    if prepared:
        v9_linear.prepare_for_prefill(Wd)
    w = (torch.rand(K, generator=torch.Generator().manual_seed(T + K)) + 0.5).half()
    y = torch.from_numpy(O.rmsnorm_fp16(X.numpy(), w.numpy(), 1e-5)).to(dev)
    assert torch.equal(v9_linear.v9_linear_forward_rmsnorm(X.to(dev), w.to(dev), 1e-5, Wd), v9_linear.v9_linear_forward(y, Wd))
    GU = synth.make_activations(T, 2 * K, seed=T + 5, outlier_frac=0.0, std=1.5)
    h = torch.from_numpy(O.silu_mul_fp16(GU[:, :K].numpy(), GU[:, K:].numpy())).to(dev)
    assert torch.equal(v9_linear.v9_linear_forward_silu_mul(GU.to(dev), Wd), v9_linear.v9_linear_forward(h, Wd))
    assert _lib.device_error(dev) == 0

"""The many-token kernel on 256-token tiles against the oracle and, bit for bit, against the 128-token one (which
callers' s8 codes select): ragged tokens and rows on both sides of a tile edge, one and many scale tables and
zero-point products (16 groups each, more of them than ring slots), residual blocks, both output layouts."""

import numpy as np
import pytest
import torch

from helpers import assert_close_fp16, container_np, make_case, np_, oracle_fused

pytestmark = pytest.mark.gpu


# shapes the library sends to the wide tiles on 148 SMs: enough block-rows that halving the tiles halves the waves
@pytest.mark.parametrize("T,N,K,density", [(257, 128 * 120, 128, 0.5), (511, 128 * 60 + 40, 384, 0.2), (255, 128 * 100 + 1, 2048, 0.0),
                                           (129, 128 * 140 + 8, 2176, 0.05), (385, 128 * 74, 9216, 0.0), (256, 128 * 75 + 4, 256, 1.0)])
@pytest.mark.parametrize("prepared", [False, True])
def test_wide_tiles_equal_narrow_tiles_and_oracle(T, N, K, density, prepared):
    from zip_kernel_b200 import _lib, ops
    W, X = make_case(T, N, K, density, perm_seed=5)
    Wd = W.to(torch.device("cuda"))
    q = ops.activation_quant_cuda(X.cuda(), Wd.perm)
    base = (Wd.W_low_packed, Wd.W_high_blocks_packed, Wd.hp_row_offsets, Wd.hp_col_indices)
    prep = (ops.prepare_weights_cuda(base[0]), ops.prepare_weights_cuda(base[1])) if prepared else None
    XE, sumxf = ops.expand_activations_cuda(q[0], q[2])
    Yn = ops.fused_dense_sparse_expanded_cuda(*base, XE, sumxf, Wd.scale_u4, Wd.zero_u4, q[1], N, K, force="tensor")
    args = (*base, q[0], Wd.scale_u4, Wd.zero_u4, q[2], q[1], N, K)
    Y = ops.fused_dense_sparse_cuda(*args, force="tensor", prepared=prep)
    assert torch.equal(Y, Yn)
    Yt = ops.fused_dense_sparse_cuda(*args, force="tensor", prepared=prep, token_major=True)
    assert torch.equal(Yt.t(), Yn)
    assert _lib.device_error(torch.device("cuda")) == 0
    # the last block-row (ragged for most shapes) against the oracle
    Wn, r0 = container_np(W), (N - 1) // 128 * 128
    b0 = int(Wn["hp_row_offsets"][-2])
    sub = dict(Wn, W_low_packed=Wn["W_low_packed"][r0:], scale_u4=Wn["scale_u4"][r0:], zero_u4=Wn["zero_u4"][r0:], d_out=N - r0,
               W_high_blocks_packed=Wn["W_high_blocks_packed"][b0:], hp_col_indices=Wn["hp_col_indices"][b0:],
               hp_row_offsets=(Wn["hp_row_offsets"][-2:] - b0).astype(np.int32))
    xs4, sx, sumx = (np_(t) for t in q)
    assert_close_fp16(np_(Y[r0:]), oracle_fused(sub, xs4, sumx, sx), "wide tiles vs oracle")

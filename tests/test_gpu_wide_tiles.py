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
    assert ops.gemm_choice(T, N, K, Wd.n_hp_blocks, prepared=prepared, force="tensor") == (_lib.KERNEL_TILES_256, _lib.CODES_E4M3)
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


# both tiles on demand: few tokens, more token tiles than a band of the CTA order holds, residual steps that cross a scale
# table (16 steps) with vector and scalar scale loads, empty block-rows, row counts on either side of a tile edge
@pytest.mark.parametrize("T,N,K,density", [(1, 256, 256, 0.5), (16, 129, 512, 0.3), (100, 200, 384, 0.3), (128, 127, 128, 1.0),
                                           (300, 640, 1024, 1.0), (257, 384, 2048, 1.0), (130, 512, 1920, 0.6), (4300, 300, 256, 0.5),
                                           (64, 128, 4608, 0.0)])
@pytest.mark.parametrize("prepared", [False, True])
def test_both_tiles_on_demand(T, N, K, density, prepared):
    from zip_kernel_b200 import _lib, ops
    dev = torch.device("cuda")
    W, X = make_case(T, N, K, density, perm_seed=7)
    Wd, Xd = W.to(dev), X.to(dev)
    base = (Wd.W_low_packed, Wd.W_high_blocks_packed, Wd.hp_row_offsets, Wd.hp_col_indices)
    prep = (ops.prepare_weights_cuda(base[0]), ops.prepare_weights_cuda(base[1])) if prepared else None
    for force, kernel in (("tensor128", _lib.KERNEL_TILES_128), ("tensor256", _lib.KERNEL_TILES_256)):
        assert ops.gemm_choice(T, N, K, Wd.n_hp_blocks, prepared=prepared, force=force)[0] == kernel
    q = ops.activation_quant_cuda(Xd, Wd.perm)
    args = (*base, q[0], Wd.scale_u4, Wd.zero_u4, q[2], q[1], N, K)
    Yn = ops.fused_dense_sparse_cuda(*args, force="tensor128", prepared=prep)
    Yw = ops.fused_dense_sparse_cuda(*args, force="tensor256", prepared=prep)
    assert torch.equal(Yw, Yn)
    xs4, sx, sumx = (np_(t) for t in q)
    Wn = container_np(W)
    assert_close_fp16(np_(Yw), oracle_fused(Wn, xs4, sumx, sx), "both tiles vs oracle")
    for force in ("tensor128", "tensor256"):       # quantised inside the call, the other output layout
        Ye = ops.fused_dense_sparse_e2e_cuda(Xd, Wd.perm, *base, Wd.scale_u4, Wd.zero_u4, N, K, force=force, prepared=prep, token_major=True)
        assert torch.equal(Ye.t(), Yn), force
    if not prepared:
        dense = (base[0], q[0], Wd.scale_u4, Wd.zero_u4, q[2], q[1])
        assert torch.equal(ops.dense_gemm_cuda(*dense, force="tensor256"), ops.dense_gemm_cuda(*dense, force="tensor128"))
        sparse = (base[1], base[2], base[3], q[0], Wd.scale_u4, q[1], N, K)
        Yh = ops.sparse_gemm_cuda(*sparse, force="tensor256")
        assert torch.equal(Yh, ops.sparse_gemm_cuda(*sparse, force="tensor128"))
        assert_close_fp16(np_(Yh), oracle_fused(Wn, xs4, sumx, sx, dense=False, sparse_weight=1.0), "residual only")
    assert _lib.device_error(dev) == 0


def test_residual_only_call_with_an_empty_block_row():
    from zip_kernel_b200 import _lib, ops
    dev = torch.device("cuda")
    T, N, K = 300, 512, 1024
    W, X = make_case(T, N, K, 0.5)
    q = ops.activation_quant_cuda(X.to(dev), W.perm.to(dev))
    ro = W.hp_row_offsets.clone()
    b1, b2 = int(ro[1]), int(ro[2])                 # take the blocks of block-row 1 out
    ro[2:] -= b2 - b1
    hi = torch.cat([W.W_high_blocks_packed[:b1], W.W_high_blocks_packed[b2:]]).to(dev)
    ci = torch.cat([W.hp_col_indices[:b1], W.hp_col_indices[b2:]]).to(dev)
    out = [ops.sparse_gemm_cuda(hi, ro.to(dev), ci, q[0], W.scale_u4.to(dev), q[1], N, K, force=f) for f in ("tensor256", "tensor128", "stream")]
    assert torch.equal(out[0], out[1])
    assert_close_fp16(np_(out[0]), np_(out[2]), "wide tiles vs streaming kernel")
    assert not out[0][128:256].any()
    assert _lib.device_error(dev) == 0


@pytest.mark.parametrize("prepared", [False, True])
def test_full_size_gate_up_on_both_tiles(prepared):
    from zip_kernel_b200 import _lib, ops
    T, K, N = 2048, 4096, 28672
    W, X = make_case(T, N, K, 0.05, perm_seed=9)
    Wd = W.to(torch.device("cuda"))
    base = (Wd.W_low_packed, Wd.W_high_blocks_packed, Wd.hp_row_offsets, Wd.hp_col_indices)
    prep = (ops.prepare_weights_cuda(base[0]), ops.prepare_weights_cuda(base[1])) if prepared else None
    args = (X.cuda(), Wd.perm, *base, Wd.scale_u4, Wd.zero_u4, N, K)
    assert ops.gemm_choice(T, N, K, Wd.n_hp_blocks, prepared=prepared)[0] == _lib.KERNEL_TILES_256
    assert torch.equal(ops.fused_dense_sparse_e2e_cuda(*args, prepared=prep),
                       ops.fused_dense_sparse_e2e_cuda(*args, prepared=prep, force="tensor128"))
    assert _lib.device_error(torch.device("cuda")) == 0


def test_tile_flags_are_checked():
    from zip_kernel_b200 import _lib, ops
    T, N, K = 128, 256, 512
    W, X = make_case(T, N, K, 0.2)
    Wd = W.to(torch.device("cuda"))
    base = (Wd.W_low_packed, Wd.W_high_blocks_packed, Wd.hp_row_offsets, Wd.hp_col_indices)
    q = ops.activation_quant_cuda(X.cuda(), Wd.perm)
    tail = (Wd.scale_u4, Wd.zero_u4, q[1], N, K)
    for fmt in (False, "packed"):                   # codes the 256-token kernel does not read
        XE, sumxf = ops.expand_activations_cuda(q[0], q[2], e4m3=fmt)
        with pytest.raises(ValueError):
            ops.fused_dense_sparse_expanded_cuda(*base, XE, sumxf, *tail, e4m3=fmt, force="tensor256")
    with pytest.raises(ValueError):
        ops.dump_accumulators(*base, q[0], N, K, force="tensor256")
    assert _lib.load().w4a4_gemm_choice(T, K, N, 0, _lib.FLAG_TILES_128 | _lib.FLAG_TILES_256, 0) == -1
    with pytest.raises(ValueError):
        ops.gemm_choice(T, N, K, force="wide")


# (tokens, d_out, d_in, residual blocks, prepared, token-major, 256-token tiles): the measured winner on 148 SMs
@pytest.mark.parametrize("T,N,K,nnz,prepared,token_major,wide", [
    (384, 6144, 256, 5, False, True, False), (512, 4096, 512, 6, False, True, False), (512, 4096, 1024, 13, True, True, False),
    (128, 4096, 512, 6, False, True, True), (192, 4096, 256, 3, True, True, True), (384, 28672, 4096, 358, True, True, False),
    (512, 4096, 14336, 179, True, True, False), (600, 4096, 14336, 179, True, True, True), (1024, 6144, 4096, 77, False, True, False),
    (1024, 6144, 4096, 77, True, True, True), (2048, 28672, 4096, 358, False, True, True),
    (256, 4096, 4096, 51, True, False, False), (257, 4096, 4096, 51, True, False, True), (257, 4096, 4096, 51, True, True, False),
    (257, 4096, 14336, 179, False, False, False), (104, 336, 640, 1, True, False, True), (128, 336, 640, 1, True, False, False),
    (112, 592, 384, 2, False, False, True), (776, 1024, 512, 2, False, False, False)])
def test_tile_choice(T, N, K, nnz, prepared, token_major, wide):
    from zip_kernel_b200 import _lib, ops
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the expected choices are those of 148 SMs")
    want = _lib.KERNEL_TILES_256 if wide else _lib.KERNEL_TILES_128
    assert ops.gemm_choice(T, N, K, nnz, prepared=prepared, token_major=token_major, force="tensor")[0] == want


# outputs whose rows start at every remainder of 16 bytes, in both layouts and with an unaligned base; nothing around them is touched
@pytest.mark.parametrize("T,N", [(256 + r, 128 + r) for r in range(1, 9)] + [(1, 131), (2, 1), (129, 257), (8, 3), (1000, 260), (520, 129)])
@pytest.mark.parametrize("base_off", [0, 1, 4])
def test_stores_of_unaligned_rows(T, N, base_off):
    from zip_kernel_b200 import _lib, ops
    lib, dev = _lib.load(), torch.device("cuda")
    K = 256
    W, X = make_case(T, N, K, 0.3)
    Wd = W.to(dev)
    q = ops.activation_quant_cuda(X.to(dev), Wd.perm)
    ws = _lib.workspace(dev, T, K, N, Wd.n_hp_blocks)
    nnz = Wd.n_hp_blocks

    def call(flags):
        buf = torch.full((T * N + 32,), 7.0, dtype=torch.float16, device=dev)
        Y = buf[8 + base_off:8 + base_off + T * N]
        rc = lib.w4a4_fused_dense_sparse(
            Wd.W_low_packed.data_ptr(), Wd.W_high_blocks_packed.data_ptr() if nnz else None, Wd.hp_row_offsets.data_ptr(),
            Wd.hp_col_indices.data_ptr() if nnz else None, q[0].data_ptr(), Wd.scale_u4.data_ptr(), Wd.zero_u4.data_ptr(), q[2].data_ptr(),
            q[1].data_ptr(), Y.data_ptr(), T, K, N, nnz, flags | _lib.FLAG_FORCE_TENSOR, ws.data_ptr(), ws.numel(),
            torch.cuda.current_stream().cuda_stream)
        assert rc == 0, lib.w4a4_last_error()
        assert bool((buf[:8 + base_off] == 7.0).all()) and bool((buf[8 + base_off + T * N:] == 7.0).all())
        return Y
    for layout in (0, _lib.FLAG_OUT_TOKEN_MAJOR):
        assert torch.equal(call(layout | _lib.FLAG_TILES_256), call(layout | _lib.FLAG_TILES_128))
    assert _lib.device_error(dev) == 0

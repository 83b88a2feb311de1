"""The bounded wait of the 256-token kernel: it lasts at least a second of real time, whatever the hardware makes of its
suspend hint, and the time a preceding kernel takes does not count towards it."""

import ctypes

import pytest
import torch

from helpers import make_case

pytestmark = pytest.mark.gpu


def elapsed_s(fn):
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    fn()
    b.record()
    b.synchronize()
    return a.elapsed_time(b) * 1e-3


def error_word(lib, stream):
    word = ctypes.c_int(0)
    lib.w4a4_device_error(ctypes.byref(word), stream)
    return word.value


def test_suspended_wait_lasts_a_second_and_reports():
    from zip_kernel_b200 import _lib
    lib, stream = _lib.load(), torch.cuda.current_stream().cuda_stream
    assert error_word(lib, stream) == 0
    assert lib.w4a4_selftest_suspended_wait(stream) == 0            # loads the kernel
    first = error_word(lib, stream)
    dt = elapsed_s(lambda: lib.w4a4_selftest_suspended_wait(stream))
    assert first == error_word(lib, stream) == 0x40000000 | (0x7e << 8)
    assert error_word(lib, stream) == 0
    assert 1.0 <= dt < 8.0, dt


def test_a_stalled_predecessor_does_not_use_up_the_wait():
    """An output exchange whose peer never sends holds the stream until its own poll limit, for longer than the GEMM's
    waits last; the GEMM behind it, resident since the exchange started, must still give its full result."""
    from zip_kernel_b200 import _lib, ops
    lib, dev = _lib.load(), torch.device("cuda")
    T, N, K = 256, 128 * 120, 1024
    W, X = make_case(T, N, K, 0.05)
    Wd = W.to(dev)
    prep = (ops.prepare_weights_cuda(Wd.W_low_packed), ops.prepare_weights_cuda(Wd.W_high_blocks_packed))
    q = ops.activation_quant_cuda(X.to(dev), Wd.perm)
    XE, sumxf = ops.expand_activations_cuda(q[0], q[2], e4m3=True)

    def gemm():
        return ops.fused_dense_sparse_expanded_cuda(Wd.W_low_packed, Wd.W_high_blocks_packed, Wd.hp_row_offsets, Wd.hp_col_indices,
                                                    XE, sumxf, Wd.scale_u4, Wd.zero_u4, q[1], N, K, prepared=prep, e4m3=True)
    assert ops.gemm_choice(T, N, K, Wd.n_hp_blocks, prepared=True) == (_lib.KERNEL_TILES_256, _lib.CODES_E4M3)
    want = gemm()
    # both "ranks" are buffers of this GPU; nothing ever raises rank 1's flag
    src = torch.zeros(16, dtype=torch.float16, device=dev)
    full = [torch.zeros(32, dtype=torch.float16, device=dev) for _ in range(2)]
    flags = [torch.zeros(2, dtype=torch.int32, device=dev) for _ in range(2)]
    state = torch.zeros(5, dtype=torch.int32, device=dev)
    ptrs = lambda ts: (ctypes.c_void_p * 2)(*[t.data_ptr() for t in ts])
    stream = torch.cuda.current_stream().cuda_stream

    def exchange(polls):
        assert lib.w4a4_peer_push_wait(src.data_ptr(), 32, ptrs(full), ptrs(flags), 64, 0, 1, 32, 2, 0, state.data_ptr(), polls,
                                       stream) == 0, lib.w4a4_last_error()
    exchange(1000)
    polls = int(200_000 * 2.5 / elapsed_s(lambda: exchange(200_000)))       # 2.5 s
    assert polls < 2 ** 30
    error_word(lib, stream)
    out = []
    dt = elapsed_s(lambda: (exchange(polls), out.append(gemm())))
    assert 1.5 < dt < 10.0, dt
    assert (error_word(lib, stream) >> 8) & 0x7f == 0x60                    # the exchange's wait, nothing of the GEMM
    assert torch.equal(out[0], want)

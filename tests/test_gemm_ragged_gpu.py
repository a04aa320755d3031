"""Int8 products whose shapes sit on the edges of the kernels that take them: few rows (the one-launch
kernel), row lengths off the 16-byte grid and right-hand sides given as [K, N] (copies in the
workspace), operands that start off 16-byte boundaries.  Bit-exact against the CPU oracle."""
import numpy as np
import pytest
import torch

from glow_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"

SHAPES = [(1, 1, 1), (1, 15, 8), (3, 17, 9), (16, 16, 33), (17, 63, 31), (8, 65, 250), (33, 479, 40), (64, 1025, 24),
          (65, 479, 65), (129, 31, 64), (130, 145, 300), (200, 1000, 129), (70, 33, 4100), (5, 4099, 7)]


def dev(a, shift=0):
    """The array on the device, `shift` bytes behind a 16-byte boundary."""
    a = np.ascontiguousarray(a)
    buf = torch.zeros(a.nbytes + 16 + shift, dtype=torch.uint8, device=DEV)
    at = -buf.data_ptr() % 16 + shift
    view = buf[at:at + a.nbytes].view(torch.from_numpy(a).dtype).view(a.shape)
    view.copy_(torch.from_numpy(a))
    return view


@pytest.mark.parametrize("M,K,N", SHAPES)
@pytest.mark.parametrize("w_off", [0, 7])
def test_int8_products(oracle, M, K, N, w_off):
    rng = np.random.default_rng(M + 3 * K + 7 * N + w_off)
    x = rng.integers(-128, 128, (M, K)).astype(np.int8)
    w = rng.integers(-128, 128, (N, K)).astype(np.int8)
    bias = rng.integers(-2 ** 15, 2 ** 15, N).astype(np.int32)
    offs = np.full(N, w_off, np.int32) if w_off == 0 else rng.integers(-20, 20, N).astype(np.int32)
    p = ops.rowwise_requant_params(rng.uniform(0.001, 0.02, N).astype(np.float32), 0.05, np.float32(5e-4),
                                   np.float32(0.5 * np.sqrt(K / 4096.0)))
    want = oracle.rowwise_quantized_fc_i8_i32(x, w, bias, offs, p[:3], p[3:], -2, 3, 1, threads=4)
    dp = [dev(a) for a in p]
    status = ops.new_status(DEV)
    for shift in (0, 1):
        for flags in ((ops.FC_WEIGHT_OFFSETS_ZERO if w_off == 0 else 0), 0):
            got = ops.rowwise_quantized_fc(dev(x, shift), dev(w, 3 * shift), dev(bias), dev(offs), dp[:3], dp[3:], -2, 3, 1,
                                           flags=flags, status=status)
            np.testing.assert_array_equal(got.cpu().numpy(), want)
    kn = np.ascontiguousarray(w.T)
    bt = ops.quantize_scale_offset_32to8(np.float32(1.5))
    ot = ops.quantize_scale_offset_32to8(np.float32(0.004 / np.sqrt(K)))
    want = oracle.fc_i8_i32(x, kn, bias, -4, 3, w_off, 1, bt, ot, threads=4)
    want_mm = oracle.matmul_i8(x, kn, 5, -3, w_off, ot, threads=4)
    for shift in (0, 2):
        got = ops.fully_connected_i8(dev(x, shift), dev(kn, shift), dev(bias), -4, 3, w_off, 1, bt, ot, status=status)
        np.testing.assert_array_equal(got.cpu().numpy(), want)
        got = ops.matmul_i8(dev(x, shift), dev(kn, shift), 5, -3, w_off, ot, status=status)
        np.testing.assert_array_equal(got.cpu().numpy(), want_mm)
    assert int(status.item()) == 0


@pytest.mark.parametrize("M,K,N", SHAPES)
@pytest.mark.parametrize("zero_offsets", [True, False])
def test_dynamic_products(oracle, M, K, N, zero_offsets):
    rng = np.random.default_rng(M + 3 * K + 7 * N)
    x = (rng.normal(0, 1, (M, K)) * rng.uniform(0.01, 30, (M, 1))).astype(np.float16)
    w = rng.integers(-128, 128, (K, N), dtype=np.int8)
    bias, scales = rng.normal(0, 2, N).astype(np.float32), rng.uniform(0.001, 0.02, N).astype(np.float32)
    offs = np.zeros(N, np.int32) if zero_offsets else rng.integers(-20, 20, N).astype(np.int32)
    want = oracle.dynamic_rowwise_quantized_fc(x, w, bias, scales, offs)
    status = ops.new_status(DEV)
    for shift in (0, 2):
        for kw in ({}, {"weights_transposed": dev(w.T, shift)}):
            got = ops.dynamic_rowwise_quantized_fc(dev(x, shift), None if kw else dev(w, shift), dev(bias), dev(scales), dev(offs),
                                                   flags=ops.FC_WEIGHT_OFFSETS_ZERO if zero_offsets else 0, status=status, **kw)
            np.testing.assert_array_equal(got.cpu().numpy().view(np.uint16), want.view(np.uint16))
    assert int(status.item()) == 0


@pytest.mark.parametrize("M,K,N", [(300, 160, 48), (300, 33, 48), (2100, 64, 40), (8, 64, 24)])
@pytest.mark.parametrize("shift", [0, 1])
def test_workspaces_of_every_size(oracle, M, K, N, shift):
    """From the least that a [K, N] product asks for to what the library names: the same results, operands off
    16-byte boundaries included; [N, K] products run with any."""
    rng = np.random.default_rng(M + K)
    x, kn = rng.integers(-128, 128, (M, K)).astype(np.int8), rng.integers(-128, 128, (K, N)).astype(np.int8)
    ot = ops.quantize_scale_offset_32to8(np.float32(0.004 / np.sqrt(K)))
    want = oracle.matmul_i8(x, kn, 5, -3, 7, ot, threads=4)
    up = lambda v, a: (v + a - 1) // a * a
    least = up(N * 4, 256) + up(M * 4, 256) + up(N * K, 256)
    pitch = up(K, 16)
    sizes = [least, least + up(M * pitch, 256), least - up(N * K, 256) + up(N * pitch, 256) + (up(M * pitch, 256) if shift else 0),
             ops.i8_gemm_workspace_bytes(M, K, N)]
    status = ops.new_status(DEV)
    for size in sizes:
        ws = torch.full((size,), 77, dtype=torch.uint8, device=DEV)
        got = ops.matmul_i8(dev(x, shift), dev(kn, 2 * shift), 5, -3, 7, ot, workspace=ws, status=status)
        np.testing.assert_array_equal(got.cpu().numpy(), want)
    with pytest.raises(Exception, match="needed"):
        ops.matmul_i8(dev(x), dev(kn), 5, -3, 7, ot, workspace=ws[:least - 1])
    bias = rng.integers(-2 ** 15, 2 ** 15, N).astype(np.int32)
    offs = rng.integers(-20, 20, N).astype(np.int32)
    p = ops.rowwise_requant_params(rng.uniform(0.001, 0.02, N).astype(np.float32), 0.05, np.float32(5e-4), np.float32(0.1))
    want = oracle.rowwise_quantized_fc_i8_i32(x, np.ascontiguousarray(kn.T), bias, offs, p[:3], p[3:], -2, 3, 1, threads=4)
    dp = [dev(a) for a in p]
    for size in (up(N * 4, 256) + up(M * 4, 256), ops.i8_gemm_workspace_bytes(M, K, N)):
        ws = torch.full((size,), 77, dtype=torch.uint8, device=DEV)
        got = ops.rowwise_quantized_fc(dev(x, shift), dev(kn.T, 3 * shift), dev(bias), dev(offs), dp[:3], dp[3:], -2, 3, 1, workspace=ws,
                                       status=status)
        np.testing.assert_array_equal(got.cpu().numpy(), want)
    assert int(status.item()) == 0


@pytest.mark.parametrize("m,n", [(2048, 1000), (2049, 1024), (4096, 500), (4097, 512), (3136, 512), (9472, 256), (9473, 250)])
def test_products_on_either_side_of_one_round_of_tiles(m, n):
    """128-column tiles that all have an SM at once, and one more: the same integers as the loop the reference has."""
    rng = np.random.default_rng(m)
    k = 144
    x, w = (torch.from_numpy(rng.integers(-128, 128, s, dtype=np.int8)).cuda() for s in ((m, k), (n, k)))
    col = lambda lo, hi: torch.from_numpy(rng.integers(lo, hi + 1, n, dtype=np.int32)).cuda()
    args = (x, w, col(-4000, 4000), col(0, 0), (col(0, 1), col(0, 9), col(1, 90)), (col(2, 3), col(15, 15), col(255, 510)), 3, -5, 0)
    want = ops.rowwise_quantized_fc(*args, flags=ops.FC_WEIGHT_OFFSETS_ZERO | ops.FC_FORCE_ANY_SHAPE_KERNEL)
    assert torch.equal(ops.rowwise_quantized_fc(*args, flags=ops.FC_WEIGHT_OFFSETS_ZERO), want)

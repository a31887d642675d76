"""Rows of the tensor-memory kernels: matrices of few units and of many, last tiles of few rows, every row format; and the two ways Q6_K rows come in by, which
carry the same arithmetic.

Bounds: as in the tests of those kernels, 1e-3 for f16 operands with f32 outputs, 3e-3 with bf16 outputs."""
import pytest
import torch

from helpers import rel_l2
from light_b200 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["q4_k", "q6_k", "q8_0", "int4", "fp8"])
@pytest.mark.parametrize("M,N,K", [(66, 128, 256), (70, 4, 512), (128, 1284, 2048), (257, 132, 6144), (96, 19000, 2048)])
def test_many_rows(cuda, kind, M, N, K):
    g = torch.Generator(device=cuda).manual_seed(N)
    dt = torch.bfloat16 if kind in ("int4", "fp8") else torch.float32
    x = torch.randn(M, K, generator=g, device=cuda).to(dt)
    if kind == "int4":
        w4 = ops.Int4(torch.randint(-2**31, 2**31, (N, K // 8), generator=g, device=cuda, dtype=torch.int32), torch.rand(N, K // 128, generator=g, device=cuda) * 0.02,
                      torch.randint(0, 16, (N, K // 128), generator=g, device=cuda).float(), 128)
        y, w = ops.MatMulInt4(x, w4), ops.DequantizeInt4(w4, torch.bfloat16).double()
    elif kind == "fp8":
        codes, scale = synth.random_fp8_block(N + K, N, K, 4, 64, device=cuda)
        y, w = ops.MatMulF8Block(x, codes, scale, 4, 64), ops.DequantizeF8Block(codes, scale, 4, 64, torch.bfloat16).double()
    else:
        t = {"q4_k": ops.Q4_K, "q6_k": ops.Q6_K, "q8_0": ops.Q8_0}[kind]
        q = ops.QTensor(synth.gaussian_weight(N + K, t, N, K, device=cuda).reshape(-1), t, (N, K))
        y, w = ops.MatMulQ(x, q), ops.Dequantize(q).double()
    assert ops.prefill_status(0) == 0
    assert rel_l2(y.cpu().double().numpy(), (x.double() @ w.t()).cpu().numpy()) <= (1e-3 if dt == torch.float32 else 3e-3)


@pytest.mark.parametrize("M,N,K", [(18, 4100, 2048), (33, 12804, 2048), (64, 2564, 14336), (65, 388, 4096), (333, 1028, 2048)])
def test_q6_k_rows_by_tma_and_by_cp_async(cuda, M, N, K):
    """Rows of a multiple of eight blocks at a 16-byte boundary come by TMA, four bytes off one they do not: value for value the same operands, in the same order."""
    raw = synth.gaussian_weight(N + M, ops.Q6_K, N, K, device=cuda).reshape(-1)
    off = torch.empty(raw.numel() + 16, dtype=raw.dtype, device=cuda)[4:4 + raw.numel()]
    off.copy_(raw)
    assert raw.data_ptr() % 16 == 0 and off.data_ptr() % 16 == 4
    x = torch.randn(M, K, generator=torch.Generator(device=cuda).manual_seed(M), device=cuda)
    y, z = (ops.MatMulQ(x, ops.QTensor(d, ops.Q6_K, (N, K))) for d in (raw, off))
    assert ops.prefill_status(0) == 0
    assert torch.equal(y, z)
    w = ops.Dequantize(ops.QTensor(raw, ops.Q6_K, (N, K))).double()
    assert rel_l2(y.cpu().double().numpy(), (x.double() @ w.t()).cpu().numpy()) <= 1e-3


@pytest.mark.parametrize("M", [4, 8, 9, 16, 33])
@pytest.mark.parametrize("N,K", [(1024, 1024), (1020, 1280), (4100, 256), (130, 8448), (409600, 256)])
def test_few_rows_of_int4(cuda, M, N, K):
    """From 2^20 weights on (100 * 2^20: from nine rows): x in f16, then the bf16 output's rounding (2^-8 of a value at most)."""
    g = torch.Generator(device=cuda).manual_seed(N)
    w = ops.Int4(torch.randint(-2**31, 2**31, (N, K // 8), generator=g, device=cuda, dtype=torch.int32), torch.rand(N, K // 128, generator=g, device=cuda) * 0.02,
                 torch.randint(0, 16, (N, K // 128), generator=g, device=cuda).float(), 128)
    x = torch.randn(M, K, generator=g, device=cuda).bfloat16()
    y = ops.MatMulInt4(x, w)
    assert torch.equal(y, ops.MatMulInt4(x, w)) and ops.prefill_status(0) == 0
    want = x.double() @ ops.DequantizeInt4(w, torch.float32).double().t()
    assert rel_l2(y.cpu().double().numpy(), want.cpu().numpy()) <= 2.5e-3


@pytest.mark.parametrize("dt,M,N,K", [(ops.Q6_K, 9, 1024, 2048), (ops.Q6_K, 16, 1028, 3584), (ops.Q6_K, 12, 2048, 5632), (ops.Q6_K, 10, 4100, 512), (ops.Q6_K, 33, 1024, 2048),
                                      (ops.Q4_K, 33, 1024, 2048), (ops.Q4_K, 64, 1030, 4096), (ops.Q4_K, 47, 2052, 2048), (ops.Q6_K, 64, 2052, 2560), (ops.Q4_K, 40, 1024, 8192)])
def test_small_matrices_of_9_to_64_rows(cuda, dt, M, N, K):
    q = ops.QTensor(synth.gaussian_weight(N + M, dt, N, K, device=cuda).reshape(-1), dt, (N, K))
    x = torch.randn(M, K, generator=torch.Generator(device=cuda).manual_seed(K), device=cuda)
    y = ops.MatMulQ(x, q)
    assert torch.equal(y, ops.MatMulQ(x, q)) and ops.prefill_status(0) == 0
    assert rel_l2(y.cpu().double().numpy(), (x.double() @ ops.Dequantize(q).double().t()).cpu().numpy()) <= 1e-3


@pytest.mark.parametrize("kind", ["q4_k", "q8_0", "int4", "fp8"])
@pytest.mark.parametrize("M,N,K", [(70, 260, 256), (100, 4100, 768), (66, 18944, 1536), (66, 19200, 1536), (129, 9480, 768), (80, 2052, 2048)])
def test_short_rows(cuda, kind, M, N, K):
    """Tiles of fewer units than a run, of between one and two, and of two; as many as there are SMs (148), and one more."""
    test_many_rows(cuda, kind, M, N, K)


@pytest.mark.parametrize("M", [4, 8, 9, 16, 17])
@pytest.mark.parametrize("N,K", [(4096, 256), (40960, 256), (12288, 512), (8192, 512), (2560, 1792), (3072, 1536), (1024, 2304), (8192, 4096), (1792, 6912)])
def test_int4_on_both_sides_of_the_token_tiles(cuda, M, N, K):
    test_few_rows_of_int4(cuda, M, N, K)


@pytest.mark.parametrize("dt,N,K", [(ops.Q6_K, 4096, 3072), (ops.Q6_K, 3072, 4096), (ops.Q6_K, 1536, 4608), (ops.Q6_K, 1792, 4608), (ops.Q6_K, 2304, 7168), (ops.Q6_K, 2560, 7168), (ops.Q6_K, 12800, 512),
                                    (ops.Q6_K, 12288, 3072), (ops.Q4_K, 16000, 1024), (ops.Q4_K, 12800, 768), (ops.Q4_K, 16384, 512), (ops.Q4_K, 16384, 256), (ops.Q4_K, 19200, 256)])
def test_whole_numbers_on_both_sides_of_the_token_tiles(cuda, dt, N, K):
    for M in (12, 16, 48):
        test_small_matrices_of_9_to_64_rows(cuda, dt, M, N, K)

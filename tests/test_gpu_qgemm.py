"""GPU parity of the prefill GEMM (jq_qgemm through quantized_matmul with many rows).

Gate (form of dots3/ops_selftest.py:48): max |y-ref| / max|ref| <= 1e-2 and
cosine >= 0.9999 against the f64 oracle.  The kernel feeds the tensor cores weights rounded once
to the activation type, so it is also held elementwise to that model of the arithmetic:
x . round(deq(W))^T in f64, within one output rounding step plus 1e-3 of max|ref|."""
import numpy as np
import pytest
import torch

import jangq_b200 as jq
from jangq_b200 import _lib
from oracle import jang_oracle as jo

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def make_case(M, N, K, bits, gs, dtype, seed=0):
    rng = np.random.default_rng(seed)
    w = torch.from_numpy((rng.standard_normal((N, K)) * 0.02).astype(np.float32)).to(DEV).to(dtype)
    x = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float32)).to(DEV).to(dtype)
    wq, s, b = jq.quantize(w, gs, bits)
    return x, wq, s, b


def check(y, x, wq, s, b, bits, gs, dtype):
    name = "bf16" if dtype == torch.bfloat16 else "f16"
    xn = x.float().cpu().numpy().astype(np.float64)
    W = jo.dequantize_affine(wq.cpu().numpy().view(np.uint32), s.float().cpu().numpy(), b.float().cpu().numpy(),
                             bits, gs)
    ref = (xn @ W.astype(np.float64).T).astype(np.float32)
    ref_rounded = (xn @ jo.round_to(W, name).astype(np.float64).T).astype(np.float32)
    y = y.float().cpu().numpy()
    scale = np.abs(ref).max()
    assert np.abs(y - ref).max() / scale <= 1e-2
    cos = float((y.astype(np.float64) * ref).sum() / (np.linalg.norm(y.astype(np.float64)) * np.linalg.norm(ref)))
    assert cos >= 0.9999
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert np.all(np.abs(y - ref_rounded) <= ulp * np.abs(ref_rounded) + 1e-3 * scale)


@pytest.mark.parametrize("gs", (32, 64, 128))
@pytest.mark.parametrize("bits", (2, 3, 4, 5, 6, 8))
def test_qgemm_bf16_all_widths(bits, gs):
    M, N, K = 160, 200, 512
    x, wq, s, b = make_case(M, N, K, bits, gs, torch.bfloat16, seed=bits * 10 + gs)
    y = jq.quantized_matmul(x, wq, s, b, group_size=gs, bits=bits)
    assert y.shape == (M, N) and y.dtype == torch.bfloat16
    check(y, x, wq, s, b, bits, gs, torch.bfloat16)


@pytest.mark.parametrize("bits", (2, 4, 8))
def test_qgemm_f16(bits):
    x, wq, s, b = make_case(64, 128, 256, bits, 64, torch.float16, seed=bits)
    y = jq.quantized_matmul(x, wq, s, b, group_size=64, bits=bits)
    check(y, x, wq, s, b, bits, 64, torch.float16)


@pytest.mark.parametrize("M,N,K", ((17, 128, 64), (128, 128, 1024), (129, 130, 192), (512, 384, 2048),
                                   (300, 1000, 768)))
def test_qgemm_shapes(M, N, K):
    """Single k-block, exact tiles, one-past-a-tile in M and N, rows whose byte length is not a
    multiple of 16 (the store falls back to scalars), several tiles in both directions."""
    x, wq, s, b = make_case(M, N, K, 4, 64, torch.bfloat16, seed=M + N)
    y = jq.quantized_matmul(x, wq, s, b, group_size=64, bits=4)
    check(y, x, wq, s, b, 4, 64, torch.bfloat16)


def test_qgemm_leading_dims_and_canaries():
    lib = _lib.load()
    M, N, K, bits, gs = 70, 136, 256, 6, 64
    x, wq, s, b = make_case(M, N, K, bits, gs, torch.bfloat16, seed=5)
    ldx, ldy = K + 8, N + 24
    xp = torch.full((M, ldx), 9.0, dtype=torch.bfloat16, device=DEV)
    xp[:, :K] = x
    yp = torch.full((M + 2, ldy), -3.0, dtype=torch.bfloat16, device=DEV)
    _lib.check(lib.jq_qgemm(xp.data_ptr(), _lib.JQ_BF16, M, ldx, wq.data_ptr(), s.data_ptr(), b.data_ptr(),
                            _lib.JQ_BF16, N, K, bits, gs, yp.data_ptr(), _lib.JQ_BF16, ldy, _lib.stream_ptr()))
    torch.cuda.synchronize()
    check(yp[:M, :N], x, wq, s, b, bits, gs, torch.bfloat16)
    assert bool((yp[:M, N:] == -3.0).all()) and bool((yp[M:] == -3.0).all())


def test_qgemm_matches_qgemv_rows():
    """The same activation row through both kernels: the GEMM only differs by the weight rounding."""
    x, wq, s, b = make_case(48, 256, 1024, 4, 64, torch.bfloat16, seed=77)
    y_gemm = jq.quantized_matmul(x, wq, s, b, group_size=64, bits=4).float()
    y_gemv = torch.cat([jq.quantized_matmul(x[i:i + 8], wq, s, b, group_size=64, bits=4) for i in range(0, 48, 8)])
    err = (y_gemm - y_gemv.float()).abs().max() / y_gemv.float().abs().max()
    assert float(err) < 1e-2


def test_qgemm_unsupported_row_lengths():
    """K % 64 != 0, or packed rows that are not a multiple of 16 bytes: the C entry point refuses,
    quantized_matmul falls back to the general mat-vec kernel and stays correct."""
    lib = _lib.load()
    for K, bits, gs in ((96, 4, 32), (64, 3, 64)):
        x, wq, s, b = make_case(40, 64, K, bits, gs, torch.bfloat16, seed=K)
        y = torch.empty((40, 64), dtype=torch.bfloat16, device=DEV)
        rc = lib.jq_qgemm(x.data_ptr(), _lib.JQ_BF16, 40, K, wq.data_ptr(), s.data_ptr(), b.data_ptr(), _lib.JQ_BF16,
                          64, K, bits, gs, y.data_ptr(), _lib.JQ_BF16, 64, _lib.stream_ptr())
        assert rc == _lib.JQ_EUNSUPPORTED
        y = jq.quantized_matmul(x, wq, s, b, group_size=gs, bits=bits)
        ref = jo.qmatmul(x.float().cpu().numpy(), wq.cpu().numpy().view(np.uint32), s.float().cpu().numpy(),
                         b.float().cpu().numpy(), bits, gs)
        assert np.abs(y.float().cpu().numpy() - ref).max() / np.abs(ref).max() <= 1e-2


def test_device_status_clean_after_gemm():
    torch.cuda.synchronize()
    assert _lib.load().jq_device_status() == 0


@pytest.mark.parametrize("gs", (64, 128))
@pytest.mark.parametrize("bits", (2, 3, 4, 5, 6, 8))
def test_qgemm_several_row_tiles(bits, gs):
    """Five row tiles and 58 column tiles (two waves): a ragged last tile in both directions, every width and code-stage
    layout."""
    M, N, K = 1160, 7300, 384
    x, wq, s, b = make_case(M, N, K, bits, gs, torch.bfloat16, seed=bits + gs)
    y = jq.quantized_matmul(x, wq, s, b, group_size=gs, bits=bits)
    check(y, x, wq, s, b, bits, gs, torch.bfloat16)
    _lib.check(_lib.load().jq_device_status())


@pytest.mark.parametrize("bits,K", ((2, 512), (3, 384), (8, 320)))
def test_grouped_and_dense_gemm_agree_bit_for_bit(bits, K):
    """The persistent grouped kernel (one expert, tiles of 128, 192 and 256 rows) and the one-tile dense kernel, unsplit for
    fewer than sixteen k-blocks, sum the same operands in the same order."""
    from jangq_b200.moe import ExpertBank, SortedPairs, _moe_gemm
    M, N, gs = 1000, 8192, 64
    x, wq, s, b = make_case(M, N, K, bits, gs, torch.bfloat16, seed=5)
    y = jq.quantized_matmul(x, wq, s, b, group_size=gs, bits=bits)
    bank = ExpertBank(wq[None], s[None], b[None], bits, gs)
    idx = torch.zeros((M,), dtype=torch.int32, device=DEV)
    for tile_m in (128, 192, 256):
        assert torch.equal(_moe_gemm(x, SortedPairs(idx, 1, tile_m=tile_m), bank), y)


@pytest.mark.parametrize("bits", (2, 3, 4, 5, 6, 8))
@pytest.mark.parametrize("M,N,K,gs", ((200, 1000, 2048, 64), (130, 520, 4096, 128), (512, 4096, 4096, 64), (40, 300, 4480, 64)))
def test_qgemm_split_k_over_a_cluster(bits, M, N, K, gs):
    """Grids far below the SM count split K over a cluster of 2 or 4 CTAs whose accumulators meet in distributed
    shared memory: ragged rows and columns, K shares that are not equal (4480 = 70 k-blocks), every width."""
    if bits in (3, 5) and K % 128:
        K += 64
    x, wq, s, b = make_case(M, N, K, bits, gs, torch.bfloat16, seed=bits * 7 + M)
    y = jq.quantized_matmul(x, wq, s, b, group_size=gs, bits=bits)
    check(y, x, wq, s, b, bits, gs, torch.bfloat16)
    y2 = jq.quantized_matmul(x, wq, s, b, group_size=gs, bits=bits)
    assert torch.equal(y, y2)                                  # the partial sums are added in rank order
    _lib.check(_lib.load().jq_device_status())


@pytest.mark.parametrize("dtype", (torch.bfloat16, torch.float16))
@pytest.mark.parametrize("bits", (2, 3, 4, 5, 6, 8))
@pytest.mark.parametrize("M,N,K,gs,scale", (
    (17, 129, 128, 64, 0.02),      # two k-blocks: two of the four dequantizer groups stay idle; two groups per row
    (33, 257, 384, 64, 0.02),      # six groups per row: two 4-byte sidecar copies per chunk, the last one half
    (256, 128, 384, 128, 0.02),    # three groups per row: sidecars not staged; exactly one full row tile
    (257, 100, 640, 64, 0.02),     # one row past a tile, ten groups per row
    (70, 300, 2048, 128, 0.02),    # split K, one 4-byte copy per chunk
    (100, 300, 1152, 64, 4.0),     # scales above the limit of the fast expansion: the general form
    (90, 130, 256, 64, 200.0),
))
def test_qgemm_expansion_and_sidecar_forms(M, N, K, gs, scale, bits, dtype):
    """Every way scales reach the dequantizers and both register expansions, at the edges of the k-block rotation."""
    rng = np.random.default_rng(bits + M)
    w = torch.from_numpy((rng.standard_normal((N, K)) * scale).astype(np.float32)).to(DEV).to(dtype)
    x = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float32)).to(DEV).to(dtype)
    wq, s, b = jq.quantize(w, gs, bits)
    y = jq.quantized_matmul(x, wq, s, b, group_size=gs, bits=bits)
    check(y, x, wq, s, b, bits, gs, dtype)
    _lib.check(_lib.load().jq_device_status())


def round_to(v, dtype):
    """float64 -> the 16-bit type's nearest value (ties to even, subnormals), as float64.  torch goes through float32."""
    p, emin = (8, -125) if dtype == torch.bfloat16 else (11, -13)
    quantum = np.ldexp(1.0, np.maximum(np.frexp(v)[1], emin) - p)
    return np.rint(v / quantum) * quantum


@pytest.mark.parametrize("dtype", (torch.bfloat16, torch.float16))
@pytest.mark.parametrize("gs", (32, 64, 128))
@pytest.mark.parametrize("bits", (2, 3, 4, 5, 6, 8))
def test_qgemm_weight_operand_is_rounded_once(bits, gs, dtype):
    """x = identity returns the weight operand itself: rn(q * scale + bias), one rounding, bit for bit.  The expansion is
    chosen per 32 rows and k-block (the rows of a warp), so the magnitude of the scales is drawn for such blocks: all at the
    bottom of the type (float16: subnormal; bfloat16: far below one), all small, all just below the limit of the fast form, all above it, and rows on
    both sides.  The one exception, 8-bit codes with bfloat16 in the general form (groups of 32, or a scale of the warp at
    2^-5 or above), rounds to float32 first."""
    bf = dtype == torch.bfloat16
    K, N = 512, 320                                       # ten blocks of 32 rows, the last tile half full
    rng = np.random.default_rng(bits + gs)
    if bf:
        limit = {2: -1, 3: 0, 4: -5, 5: -2, 6: -3, 8: -5}[bits]
        classes = ((-100, -90), (-40, -8), (limit - 3, limit), (limit, limit + 8), (limit - 2, limit + 2))
    else:
        limit = {2: -2, 3: 0, 4: -4, 5: -2, 6: -3, 8: 4}[bits]       # 8-bit: no limit
        classes = ((-24, -14), (-14, -8), (limit - 3, limit - 0.05), (limit, limit + 3), (limit - 2, limit + 2))
    kb = max(gs, 64)
    which = rng.integers(0, len(classes), (N // 32, K // kb)).repeat(32, 0).repeat(kb // gs, 1)
    lo, hi = np.array(classes)[which].transpose(2, 0, 1)
    s = torch.from_numpy(np.exp2(rng.uniform(lo, hi)) * rng.choice([-1.0, 1.0], lo.shape)).to(DEV).to(dtype)
    sv = s.double().cpu().numpy()
    b = torch.from_numpy(sv * rng.uniform(-2.0 ** bits, 2.0, sv.shape)).to(DEV).to(dtype)
    q = rng.integers(0, 2 ** bits, (N, K))
    wq = torch.from_numpy(jo.pack_rows(q, bits).view(np.int32)).to(DEV)
    exact = q * sv.repeat(gs, 1) + b.double().cpu().numpy().repeat(gs, 1)        # 53 bits hold it
    if bf and bits == 8:
        general = np.abs(sv).reshape(N // 32, 32, K // kb, -1).max((1, 3)) >= 2.0 ** -5 if gs >= 64 else np.ones((N // 32, K // kb), bool)
        exact = np.where(general.repeat(32, 0).repeat(kb, 1), exact.astype(np.float32).astype(np.float64), exact)
    y = jq.quantized_matmul(torch.eye(K, dtype=dtype, device=DEV), wq, s, b, group_size=gs, bits=bits)
    assert np.array_equal(y.double().cpu().numpy().T, round_to(exact, dtype))
    _lib.check(_lib.load().jq_device_status())


@pytest.mark.parametrize("M", (16, 17))
@pytest.mark.parametrize("bits,K", ((8, 34 << 20), (6, 46 << 20)))
def test_rows_of_34_megabytes(bits, K, M):
    """127 packed rows span more than 2^32 bytes: the last rows of a 128-row tile are the ones of their own product, bit
    for bit (both take the same K split), in the GEMM and in the small-batch mat-vec."""
    gs, N = 128, 128
    gen = torch.Generator(device=DEV)
    gen.manual_seed(bits)
    wq = torch.randint(-2 ** 31, 2 ** 31 - 1, (N, K * bits // 32), generator=gen, device=DEV, dtype=torch.int32)
    s = torch.rand((N, K // gs), generator=gen, device=DEV).bfloat16() * 1e-4
    b = -s
    x = torch.empty((M, K), dtype=torch.bfloat16, device=DEV).normal_(generator=gen)
    y = jq.quantized_matmul(x, wq, s, b, group_size=gs, bits=bits)
    assert torch.equal(y[:, 96:], jq.quantized_matmul(x, wq[96:], s[96:], b[96:], group_size=gs, bits=bits))
    _lib.check(_lib.load().jq_device_status())

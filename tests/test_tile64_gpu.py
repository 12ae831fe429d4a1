"""GPU tests of the 128 x 64 GEMM tile at its edges: rows and columns that fill no tile, fewer K tiles than ring stages and more,
K parts, and every output and operand type.  Tolerance as in test_gemm_gpu.py."""
import numpy as np
import pytest

from catccos_b200 import workloads
from conftest import to_dev_bf16

pytestmark = pytest.mark.gpu


@pytest.fixture()
def tile64(capi, cuda):
    capi.set_option("small_tile", 2)
    capi.set_option("cta_pair", 2)
    capi.set_option("block_n", 64)
    yield capi
    for key in ("small_tile", "cta_pair", "block_n", "split_k", "c_dtype", "a_dtype", "b_lsu"):
        capi.set_option(key, 0)


def _problem(oracle, m, n, k):
    rng = np.random.default_rng(m + 3 * n + k)
    x = workloads.f32_to_bf16_bits(rng.standard_normal((m, k), dtype=np.float32))
    w = workloads.f32_to_bf16_bits(rng.standard_normal((k, n), dtype=np.float32) * np.float32(0.02))
    return x, (*oracle.quantize_rows(x), *oracle.quantize_weight(w))


@pytest.mark.parametrize("b_lsu", [1, 2])  # the weight by the load/store units, or by TMA
@pytest.mark.parametrize("split_k", [1, 2])
@pytest.mark.parametrize("m,n,k", [(1, 16, 128), (128, 64, 1024), (129, 80, 1152), (300, 272, 2048), (509, 528, 3968), (2000, 1040, 256)])
def test_shapes(tile64, cuda, oracle, m, n, k, split_k, b_lsu):
    _, ops = _problem(oracle, m, n, k)
    gold = oracle.allgather_matmul([ops[0]], [ops[1]], ops[2], ops[3])
    dev = [cuda.from_numpy(v).cuda() for v in ops]
    tile64.set_option("split_k", split_k)
    tile64.set_option("b_lsu", b_lsu)
    out = tile64.mx_gemm(*dev)
    bad, most = oracle.check_close(out.float().cpu().numpy(), gold, 1e-2, 1e-3)
    assert bad == 0, (bad, most)
    tile64.set_option("c_dtype", 1)
    half = tile64.mx_gemm(*dev, out_dtype=cuda.float16)
    # the same sums rounded to 11 and to 8 significant bits
    assert cuda.all((half.float() - out.float()).abs() <= 2.0 ** -8 * half.float().abs().clamp_min(2.0 ** -14))


@pytest.mark.parametrize("m,n,k", [(200, 96, 1024), (130, 544, 384)])
def test_quantised_output(tile64, cuda, oracle, m, n, k):
    _, ops = _problem(oracle, m, n, k)
    dev = [cuda.from_numpy(v).cuda() for v in ops]
    plain = tile64.mx_gemm(*dev)
    codes, scales = tile64.mx_gemm_quant_out(*dev)
    want_c, want_s = oracle.quantize_rows(plain.view(cuda.int16).cpu().numpy().view(np.uint16))
    assert np.array_equal(codes.cpu().numpy(), want_c)
    assert np.array_equal(scales.cpu().numpy(), want_s)


def test_fp4_operands(tile64, cuda, oracle):
    m, n, k = 150, 256, 1152
    ap, asc = tile64.mx_quant_fp4(to_dev_bf16(cuda, _problem(oracle, m, 16, k)[0]))
    bt, bts = tile64.mx_quant_fp4(to_dev_bf16(cuda, _problem(oracle, n, 16, k)[0]))
    values = cuda.stack((bt & 15, bt >> 4), dim=2).view(n, k).t()
    b = (values[:, 0::2] | (values[:, 1::2] << 4)).contiguous()
    bs = bts.view(n, k // 64, 2).permute(1, 0, 2).contiguous()
    out = []
    for width in (64, 128):
        tile64.set_option("block_n", width)
        c = cuda.empty((m, n), dtype=cuda.bfloat16, device="cuda")
        tile64.fp4_mx_allgather_matmul(ap, asc, b, bs, c, 0, 1)
        out.append(c.float())
    # one summation order or another, each rounded once to 8 bits
    assert cuda.all((out[0] - out[1]).abs() <= 2.0 ** -7 * out[1].abs().clamp_min(1.0))

"""GPU tests of the small-tile GEMM where it can go wrong: activation rows around its tile heights (16, 32), K parts
that do not divide the K tiles or leave one each, output columns that fill no tile, every output and operand type, and the
quantisation inside the kernel against the quantiser in front of it.  Tolerances as in test_gemm_gpu.py."""
import numpy as np
import pytest

from catccos_b200 import workloads
from conftest import to_dev_bf16

pytestmark = pytest.mark.gpu


@pytest.fixture()
def small(capi, cuda):
    capi.finalize()
    capi.set_option("small_tile", 1)
    yield capi
    for key in ("small_tile", "small_quant", "split_k", "a_dtype", "c_dtype", "b_dtype", "tiny_block_rule"):
        capi.set_option(key, 0)
    assert capi.last_status()[0] in (0, -2)  # -2: only the allocation-free path ran, which creates no rank context
    capi.finalize()


def _problem(oracle, m, n, k):
    rng = np.random.default_rng(m * 7 + n + k)
    x = workloads.f32_to_bf16_bits(rng.standard_normal((m, k), dtype=np.float32))
    w = workloads.f32_to_bf16_bits(rng.standard_normal((k, n), dtype=np.float32) * np.float32(0.02))
    return x, oracle.quantize_weight(w)


def _check(oracle, out, gold):
    bad, most = oracle.check_close(out.float().cpu().numpy(), gold, 1e-2, 1e-3)
    assert bad == 0, (bad, most)


@pytest.mark.parametrize("split_k", [0, 1, 2, 4])
@pytest.mark.parametrize("m,n,k", [(1, 16, 128), (16, 272, 1024), (17, 128, 3968), (33, 1040, 384), (64, 2304, 896), (65, 144, 1280),
                                   (128, 512, 640), (129, 256, 2304), (300, 528, 1152)])
def test_gemm_and_fused(small, cuda, oracle, m, n, k, split_k):
    torch = cuda
    x, (bc, bsc) = _problem(oracle, m, n, k)
    ac, asc = oracle.quantize_rows(x)
    gold = oracle.allgather_matmul([ac], [asc], bc, bsc)
    dev = [torch.from_numpy(v).cuda() for v in (ac, asc, bc, bsc)]
    small.set_option("split_k", split_k)
    plain = small.mx_gemm(*dev)
    _check(oracle, plain, gold)
    x_d = to_dev_bf16(torch, x)
    symm = small.symm_alloc(small.symm_bytes_needed(small.make_tiling(m, k, n, 1), False))
    for quant in (1, 2):
        small.set_option("small_quant", quant)
        c = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
        small.mx_quant_allgather_matmul(x_d, dev[2], dev[3], c, symm, 1)
        static = torch.full_like(c, float("nan"))
        small.mx_quant_matmul_static(x_d, dev[2], dev[3], static)
        assert torch.equal(static, c)
        if split_k != 0:
            assert torch.equal(c, plain)  # the same codes and scales, the same number of K parts, so the same order of summation
        else:
            _check(oracle, c, gold)  # a quantising launch may choose other K parts: another order of summation
        assert small.static_status()[0] == 0


@pytest.mark.parametrize("m,n,k", [(5, 32, 512), (40, 160, 1024), (100, 544, 384), (200, 256, 2048)])
def test_quantised_output(small, cuda, oracle, m, n, k):
    torch = cuda
    x, (bc, bsc) = _problem(oracle, m, n, k)
    dev = [torch.from_numpy(v).cuda() for v in (*oracle.quantize_rows(x), bc, bsc)]
    plain = small.mx_gemm(*dev)
    codes, scales = small.mx_gemm_quant_out(*dev)
    want_c, want_s = oracle.quantize_rows(plain.view(torch.int16).cpu().numpy().view(np.uint16))
    assert np.array_equal(codes.cpu().numpy(), want_c)
    assert np.array_equal(scales.cpu().numpy(), want_s)


@pytest.mark.parametrize("m", [7, 50, 120])
def test_types(small, cuda, oracle, m):
    torch = cuda
    n, k = 256, 1152
    x, (bc, bsc) = _problem(oracle, m, n, k)
    x_d, b_d, bs_d = to_dev_bf16(torch, x), torch.from_numpy(bc).cuda(), torch.from_numpy(bsc).cuda()
    # fp16 result and E5M2 activations, quantised inside and in front
    small.set_option("a_dtype", 1)
    small.set_option("c_dtype", 1)
    codes, scales = small.mx_quant(x_d)
    small.set_option("split_k", 2)  # the same order of summation whoever quantises
    want = small.mx_gemm(codes, scales, b_d, bs_d, out_dtype=torch.float16)
    for quant in (1, 2):
        small.set_option("small_quant", quant)
        got = torch.empty_like(want)
        small.mx_quant_matmul_static(x_d, b_d, bs_d, got)
        assert torch.equal(got, want), quant
    small.set_option("small_quant", 0)
    small.set_option("split_k", 0)
    small.set_option("small_tile", 2)
    other = small.mx_gemm(codes, scales, b_d, bs_d, out_dtype=torch.float16)
    # two fp32 summation orders, each rounded once to 11 bits: one unit in the last place of the larger
    assert torch.all((got.float() - other.float()).abs() <= 2.0 ** -10 * other.float().abs().clamp_min(1.0))
    small.set_option("small_tile", 1)
    # packed E2M1 operands
    small.set_option("a_dtype", 0)
    small.set_option("c_dtype", 0)
    ap, asc = small.mx_quant_fp4(x_d)
    bt, bts = small.mx_quant_fp4(to_dev_bf16(torch, np.ascontiguousarray(_problem(oracle, n, 16, k)[0])))
    values = torch.stack((bt & 15, bt >> 4), dim=2).view(n, k).t()
    b4 = (values[:, 0::2] | (values[:, 1::2] << 4)).contiguous()
    b4s = bts.view(n, k // 64, 2).permute(1, 0, 2).contiguous()
    out = [torch.empty((m, n), dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    for c, tile in zip(out, (1, 2)):
        small.set_option("small_tile", tile)
        small.fp4_mx_allgather_matmul(ap, asc, b4, b4s, c, 0, 1)
    assert torch.all((out[0].float() - out[1].float()).abs() <= 2.0 ** -7 * out[1].float().abs().clamp_min(1.0))


@pytest.mark.parametrize("split_k", [1, 4])
@pytest.mark.parametrize("m", [12, 40])
def test_nonfinite_blocks(small, cuda, oracle, m, split_k):
    # an infinity or a NaN makes its block NaN (code 0x7F, scale 0xFF), and with it exactly its row of the product
    torch = cuda
    n, k = 160, 2048
    x, (bc, bsc) = _problem(oracle, m, n, k)
    bad = {3: (5, 0x7F80), 6: (1024, 0xFF80), 11: (2047, 0x7FC0)}  # row: column, +inf, -inf, NaN
    rows = np.array([r for r in range(m) if r not in bad])
    ac, asc = oracle.quantize_rows(np.ascontiguousarray(x[rows]))
    gold = oracle.allgather_matmul([ac], [asc], bc, bsc)
    for r, (col, bits) in bad.items():
        x[r, col] = bits
    x_d, b_d, bs_d = to_dev_bf16(torch, x), torch.from_numpy(bc).cuda(), torch.from_numpy(bsc).cuda()
    keep, gone = torch.from_numpy(rows).cuda(), torch.tensor(sorted(bad), device="cuda")
    small.set_option("split_k", split_k)
    for quant in (1, 2):
        small.set_option("small_quant", quant)
        c = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
        small.mx_quant_matmul_static(x_d, b_d, bs_d, c)
        assert bool(c[gone].isnan().all())
        _check(oracle, c[keep], gold)
    codes, scales = small.mx_gemm_quant_out(*small.mx_quant(x_d), b_d, bs_d)
    assert bool((codes[gone] == 0x7F).all()) and bool((scales[gone] == 0xFF).all())
    want = oracle.quantize_rows(c.view(torch.int16).cpu().numpy().view(np.uint16)[rows])
    assert np.array_equal(codes[keep].cpu().numpy(), want[0]) and np.array_equal(scales[keep].cpu().numpy(), want[1])


def test_tiny_blocks(small, cuda, oracle, golden):
    # the edge fixture's zeros, subnormals, ties and tiny blocks through the quantisation inside the kernel, both rules
    torch = cuda
    x = np.ascontiguousarray(golden("quant_edges")["x"].reshape(-1)[: 128 * 24].reshape(24, 128))
    bc, bsc = _problem(oracle, 1, 32, 128)[1]
    b_d, bs_d = torch.from_numpy(bc).cuda(), torch.from_numpy(bsc).cuda()
    for rule in (0, 1):
        small.set_option("tiny_block_rule", rule)
        out = []
        for quant in (1, 2):
            small.set_option("small_quant", quant)
            c = torch.zeros((24, 32), dtype=torch.bfloat16, device="cuda")
            small.mx_quant_matmul_static(to_dev_bf16(torch, x), b_d, bs_d, c)
            out.append(c.view(torch.int16))
        assert torch.equal(*out)

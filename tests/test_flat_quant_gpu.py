"""GPU tests of the flat quantisers where their tiling has edges: a warp takes 512 values and a block of the grid 4096,
whatever the rows are, so the counts sit around those; inputs aligned to 16 bytes only take another load."""
import numpy as np
import pytest

from catccos_b200 import workloads
from conftest import to_dev_bf16

pytestmark = pytest.mark.gpu

SHAPES = [(15, 32), (16, 32), (17, 32), (127, 32), (128, 32), (129, 32), (8, 512), (7, 544), (1, 8224), (513, 4064)]


def _bits(rows, k):
    rng = np.random.default_rng(rows * 131 + k)
    return workloads.f32_to_bf16_bits(rng.standard_normal((rows, k), dtype=np.float32) * np.float32(2.0))


def _at_16_bytes(torch, bits):
    flat = torch.empty(bits.size + 8, dtype=torch.bfloat16, device="cuda")
    x = flat[8:].view(bits.shape)
    assert x.data_ptr() % 32 == 16
    x.copy_(to_dev_bf16(torch, bits))
    return x


@pytest.mark.parametrize("rows,k", SHAPES)
@pytest.mark.parametrize("half_aligned", [False, True])
def test_codes_and_scales(capi, cuda, oracle, rows, k, half_aligned):
    bits = _bits(rows, k)
    x = _at_16_bytes(cuda, bits) if half_aligned else to_dev_bf16(cuda, bits)
    want_c, want_s = oracle.quantize_rows(bits)
    codes, scales = capi.mx_quant(x)
    assert np.array_equal(codes.cpu().numpy(), want_c)
    assert np.array_equal(scales.cpu().numpy(), want_s)
    capi.set_option("tiny_block_rule", 1)
    try:
        want_p, want_s = oracle.quantize_rows_e2m1(bits, oracle.MODE_DEVICE)
        packed, scales = capi.mx_quant_fp4(x)
    finally:
        capi.set_option("tiny_block_rule", 0)
    assert np.array_equal(packed.cpu().numpy(), want_p)
    assert np.array_equal(scales.cpu().numpy(), want_s)


@pytest.mark.parametrize("tokens,n,top_k", [(1, 480, 1), (9, 512, 8), (8, 544, 3), (3, 1056, 33), (5, 64, 40)])
def test_packed_rows(capi, cuda, oracle, tokens, n, top_k):
    torch = cuda
    bits = _bits(tokens, n)
    rng = np.random.default_rng(n)
    idx = rng.permutation(tokens * top_k).astype(np.int32).reshape(tokens, top_k)
    idx[rng.random(idx.shape) < 0.1] = -1
    row_bytes = capi.packed_row_bytes(n)
    out = torch.full((tokens * top_k, row_bytes), 0xAA, dtype=torch.uint8, device="cuda")
    capi.mx_quant_scatter_packed(to_dev_bf16(torch, bits), torch.from_numpy(idx).cuda(), out, top_k)
    want = np.full((tokens * top_k, row_bytes), 0xAA, np.uint8)
    wc, ws = oracle.quantize_rows(bits)
    for t in range(tokens):
        for dst in idx[t][idx[t] >= 0]:
            want[dst] = np.concatenate([wc[t], ws[t], np.zeros(row_bytes - n - n // 32, np.uint8)])
    assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("offset", [0, 4, 1])
def test_single_rank_operands_in_place_or_through_the_stage(capi, cuda, oracle, offset):
    # quantised activations of one rank are read where they are when their scales are word-aligned, else copied first
    torch = cuda
    m, n, k = 200, 272, 384
    rng = np.random.default_rng(5)
    ac, asc = oracle.quantize_rows(_bits(m, k))
    bc, bsc = oracle.quantize_weight(workloads.f32_to_bf16_bits(rng.standard_normal((k, n), dtype=np.float32) * np.float32(0.02)))
    flat = torch.zeros(asc.size + 16, dtype=torch.uint8, device="cuda")
    scales = flat[offset:offset + asc.size].view(asc.shape)
    scales.copy_(torch.from_numpy(asc))
    c = torch.zeros((m, n), dtype=torch.bfloat16, device="cuda")
    symm = capi.symm_alloc(capi.symm_bytes_needed(capi.make_tiling(m, k, n, 1), False))
    try:
        capi.fp8_mx_allgather_matmul(torch.from_numpy(ac).cuda(), scales, torch.from_numpy(bc).cuda(), torch.from_numpy(bsc).cuda(),
                                     c, symm, 1)
        torch.cuda.synchronize()
    finally:
        capi.symm_free(symm)
    gold = oracle.allgather_matmul([ac], [asc], bc, bsc)
    bad, most = oracle.check_close(c.float().cpu().numpy(), gold, 1e-2, 1e-3)
    assert bad == 0, most

"""GPU test of one-rank calls whose output lies in the activations' memory: the result is that of a call with buffers of its
own, bit for bit (the same codes through the same tiling)."""
import numpy as np
import pytest

from catccos_b200 import workloads
from conftest import to_dev_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("small_tile", [1, 2])
@pytest.mark.parametrize("m,n,k", [(16, 1024, 1024), (300, 1040, 2048)])
def test_output_over_the_activations(capi, cuda, oracle, m, n, k, small_tile):
    torch = cuda
    rng = np.random.default_rng(m + n + k)
    x = workloads.f32_to_bf16_bits(rng.standard_normal((m, k), dtype=np.float32))
    w = workloads.f32_to_bf16_bits(rng.standard_normal((k, n), dtype=np.float32) * np.float32(0.02))
    b, b_scales = (torch.from_numpy(v).cuda() for v in oracle.quantize_weight(w))
    x_d = to_dev_bf16(torch, x)
    a, a_scales = (torch.from_numpy(v).cuda() for v in oracle.quantize_rows(x))
    symm = capi.symm_alloc(capi.symm_bytes_needed(capi.make_tiling(m, k, n, 1), False))
    capi.set_option("small_tile", small_tile)
    capi.set_option("small_quant", 1)
    capi.set_option("split_k", 4 if small_tile == 1 else 1)  # the sums of both calls run in the same order
    try:
        want = torch.empty((m, n), dtype=torch.bfloat16, device="cuda")
        capi.fp8_mx_allgather_matmul(a, a_scales, b, b_scales, want, symm, 1)
        # bf16 activations, C over their first bytes
        pool = torch.zeros(max(m * k, m * n), dtype=torch.bfloat16, device="cuda")
        shared = pool[: m * k].view(m, k)
        shared.copy_(x_d)
        c = pool[: m * n].view(m, n)
        capi.mx_quant_allgather_matmul(shared, b, b_scales, c, symm, 1)
        assert torch.equal(c, want)
        # quantised activations: codes, then scales, inside C
        raw = torch.zeros(max(2 * m * n, m * k + m * k // 32), dtype=torch.uint8, device="cuda")
        codes, scales = raw[: m * k].view(m, k), raw[m * k: m * k + m * k // 32].view(m, k // 32)
        codes.copy_(a)
        scales.copy_(a_scales)
        c = raw[: 2 * m * n].view(torch.bfloat16).view(m, n)
        capi.fp8_mx_allgather_matmul(codes, scales, b, b_scales, c, symm, 1)
        assert torch.equal(c, want)
        assert capi.last_status()[0] == 0
    finally:
        for key in ("small_tile", "small_quant", "split_k"):
            capi.set_option(key, 0)
        capi.symm_free(symm)

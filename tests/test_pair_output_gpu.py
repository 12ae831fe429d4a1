"""GPU test of how a CTA pair's tiles leave: the last tile of a pair through the operand stages, earlier ones through one buffer.
Tolerance as in test_gemm_gpu.py."""
import numpy as np
import pytest

from catccos_b200 import workloads

pytestmark = pytest.mark.gpu


# a tile cut in both directions, one column group past half a tile, one full tile, and more tiles than the GPU has pairs
@pytest.mark.parametrize("f16", [False, True])
@pytest.mark.parametrize("m,n,k", [(70, 48, 128), (256, 144, 1152), (256, 256, 128), (2570, 2320, 256)])
def test_every_tile_arrives(capi, cuda, oracle, m, n, k, f16):
    rng = np.random.default_rng(m + n + k)
    x = workloads.f32_to_bf16_bits(rng.standard_normal((m, k), dtype=np.float32))
    w = workloads.f32_to_bf16_bits(rng.standard_normal((k, n), dtype=np.float32) * np.float32(0.02))
    ops = (*oracle.quantize_rows(x), *oracle.quantize_weight(w))
    gold = oracle.allgather_matmul([ops[0]], [ops[1]], ops[2], ops[3])
    dev = [cuda.from_numpy(v).cuda() for v in ops]
    dtype = cuda.float16 if f16 else cuda.bfloat16
    out = cuda.full((m + 1, n), -77.0, dtype=dtype, device="cuda")  # the row after the last is not the call's
    try:
        for key, value in (("cta_pair", 1), ("split_k", 1), ("small_tile", 2), ("c_dtype", int(f16))):
            capi.set_option(key, value)
        capi.mx_gemm(*dev, out=out[:m], out_dtype=dtype)
    finally:
        for key in ("cta_pair", "split_k", "small_tile", "c_dtype"):
            capi.set_option(key, 0)
    bad, most = oracle.check_close(out[:m].float().cpu().numpy(), gold, 1e-2, 1e-3)
    assert bad == 0, (bad, most)
    assert bool((out[m] == -77.0).all())

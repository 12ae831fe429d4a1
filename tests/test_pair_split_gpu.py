"""GPU test of CTA pairs that begin with a part of a split tile and go on with whole ones: 76 tiles on 74 pairs, the last two cut
along K.  Those two lie at both edges of the matrix, so some warps have no rows and some chunks no columns.
Tolerance as in test_gemm_gpu.py; another order of the fp32 sums moves a bf16 result by one rounding, 2^-7 of it at most."""
import numpy as np
import pytest

from catccos_b200 import workloads

pytestmark = pytest.mark.gpu

RTOL, ATOL = 1e-2, 1e-3
OPTIONS = ("cta_pair", "small_tile", "split_k", "c_dtype")


@pytest.fixture()
def pairs(capi, cuda):
    capi.set_option("cta_pair", 1)
    capi.set_option("small_tile", 2)
    yield capi
    for key in OPTIONS:
        capi.set_option(key, 0)
    assert capi.last_status()[0] == 0


def _operands(cuda, oracle, m, n, k, seed):
    rng = np.random.default_rng(seed)
    x = workloads.f32_to_bf16_bits(rng.standard_normal((m, k), dtype=np.float32))
    w = workloads.f32_to_bf16_bits(rng.standard_normal((k, n), dtype=np.float32) * np.float32(0.02))
    ops = (*oracle.quantize_rows(x), *oracle.quantize_weight(w))
    return ops, [cuda.from_numpy(v).cuda() for v in ops]


@pytest.mark.parametrize("f16", [False, True])
def test_result(pairs, cuda, oracle, f16):
    m, n, k = 4800, 1008, 2048
    rows = np.r_[0:32, 1150:1160, 4608:4800]  # the split tiles' rows among them
    dtype = cuda.float16 if f16 else cuda.bfloat16
    pairs.set_option("c_dtype", int(f16))
    for seed in (1, 2):  # the second set meets the first one's partial tiles and flags
        ops, dev = _operands(cuda, oracle, m, n, k, seed)
        gold = oracle.allgather_matmul([ops[0][rows]], [ops[1][rows]], ops[2], ops[3])
        pairs.set_option("split_k", 1)
        whole = pairs.mx_gemm(*dev, out_dtype=dtype).float()
        for split_k in (0, 2, 3, 8):
            pairs.set_option("split_k", split_k)
            out = cuda.full((m + 1, n), -77.0, dtype=dtype, device="cuda")
            pairs.mx_gemm(*dev, out=out[:m])
            bad, most = oracle.check_close(out[:m][cuda.from_numpy(rows).cuda()].float().cpu().numpy(), gold, RTOL, ATOL)
            assert bad == 0, (split_k, bad, most)
            assert bool(((out[:m].float() - whole).abs() <= RTOL * whole.abs() + ATOL).all()), split_k
            assert bool((out[m] == -77.0).all())


def test_quantised_output(pairs, cuda, oracle):
    for seed in (3, 4):
        dev = _operands(cuda, oracle, 4800, 992, 2048, seed)[1]
        for split_k in (0, 2, 3, 8):
            pairs.set_option("split_k", split_k)
            want = pairs.mx_quant(pairs.mx_gemm(*dev))  # the same order of summation, then the quantiser
            got = pairs.mx_gemm_quant_out(*dev)
            assert cuda.equal(got[0], want[0]) and cuda.equal(got[1], want[1]), split_k

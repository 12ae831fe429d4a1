"""GPU test of one-rank calls captured in a CUDA graph: every replay works on the inputs it finds, also where K is split and the
parts of a tile wait for one another's flags.  The graph and an eager call run the same launches, so their results are equal."""
import numpy as np
import pytest

from catccos_b200 import workloads
from conftest import to_dev_bf16

pytestmark = pytest.mark.gpu

OPTIONS = ("cta_pair", "block_n", "small_tile", "split_k")
# one CTA a part; every tile of the pairs split; split tiles with whole ones behind them; no split; cluster parts
TILINGS = [
    (300, 528, 2048, dict(cta_pair=2, block_n=128, small_tile=2, split_k=4)),
    (1024, 2304, 3584, dict(cta_pair=1, small_tile=2)),
    (2400, 2080, 4096, dict(cta_pair=1, small_tile=2)),
    (512, 528, 1024, dict(cta_pair=2, small_tile=2, split_k=1)),
    (40, 528, 2048, dict(small_tile=1, split_k=4)),
]


@pytest.mark.parametrize("m,n,k,options", TILINGS)
def test_replays(capi, cuda, oracle, m, n, k, options):
    torch = cuda
    rng = np.random.default_rng(m + n + k)
    sets = []
    for _ in range(3):
        x = to_dev_bf16(torch, workloads.f32_to_bf16_bits(rng.standard_normal((m, k), dtype=np.float32)))
        w = to_dev_bf16(torch, workloads.f32_to_bf16_bits(rng.standard_normal((n, k), dtype=np.float32) * np.float32(0.02)))
        codes, scales = capi.mx_quant(w)
        sets.append((x, *capi.mx_quant(x), codes.t().contiguous(), scales.view(n, k // 64, 2).permute(1, 0, 2).contiguous()))
    symm = capi.symm_alloc(capi.symm_bytes_needed(capi.make_tiling(m, k, n, 1), False))
    for key, value in options.items():
        capi.set_option(key, value)

    def step(x, a, a_scales, b, b_scales, out):
        capi.mx_gemm(a, a_scales, b, b_scales, out=out[0])
        capi.mx_quant_allgather_matmul(x, b, b_scales, out[1], symm, 1)
        capi.fp8_mx_allgather_matmul(a, a_scales, b, b_scales, out[2], symm, 1)

    def outputs():
        return [torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(3)]

    try:
        want = []
        for s in sets:
            want.append(outputs())
            step(*s, want[-1])
        held, out = [t.clone() for t in sets[0]], outputs()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            step(*held, out)
        got = []
        for i in (0, 1, 2, 1, 0):  # nothing waits in between: each replay meets what the one before left
            for h, t in zip(held, sets[i]):
                h.copy_(t)
            graph.replay()
            got.append((i, [o.clone() for o in out]))
            if i == 2:
                step(*sets[0], outputs())  # an eager call between two replays
        torch.cuda.synchronize()
        for i, o in got:
            for a, b in zip(o, want[i]):
                assert torch.equal(a, b), i
        assert capi.last_status()[0] == 0
    finally:
        for key in OPTIONS:
            capi.set_option(key, 0)
        capi.symm_free(symm)


@pytest.mark.parametrize("small_tile", [1, 2])  # one launch, two launches
def test_replays_of_the_allocation_free_call(capi, cuda, small_tile):
    torch = cuda
    m, n, k = 48, 272, 1024
    gen = torch.Generator(device="cuda").manual_seed(1)
    xs = [torch.randn((m, k), generator=gen, device="cuda").to(torch.bfloat16) for _ in range(3)]
    codes, scales = capi.mx_quant((torch.randn((n, k), generator=gen, device="cuda") * 0.02).to(torch.bfloat16))
    b, b_scales = codes.t().contiguous(), scales.view(n, k // 64, 2).permute(1, 0, 2).contiguous()
    capi.set_option("small_tile", small_tile)
    capi.set_option("small_quant", small_tile)
    try:
        want = []
        for x in xs:
            want.append(torch.empty((m, n), dtype=torch.bfloat16, device="cuda"))
            capi.mx_quant_matmul_static(x, b, b_scales, want[-1])
        x, c = xs[0].clone(), torch.empty_like(want[0])
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            capi.mx_quant_matmul_static(x, b, b_scales, c)
            capi.mx_quant_matmul_static(x, b, b_scales, c)
        for i in (0, 1, 2, 1):
            x.copy_(xs[i])
            c.fill_(float("nan"))
            graph.replay()
            other = torch.empty_like(c)
            capi.mx_quant_matmul_static(xs[0], b, b_scales, other)
            assert torch.equal(c, want[i]) and torch.equal(other, want[0])
            assert capi.static_status()[0] == 0
    finally:
        capi.set_option("small_tile", 0)
        capi.set_option("small_quant", 0)

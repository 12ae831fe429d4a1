"""GPU test of the device-side timeline (trace build): every one-rank call leaves one, also where the product build would take
the small-tile kernel, which keeps none."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import torch
from catccos_b200 import capi, timeline

assert capi.TRACE
for m, n, k in ((16, 1024, 1024), (1024, 2304, 1024)):
    x = torch.randn((m, k), device="cuda").to(torch.bfloat16)
    codes, scales = capi.mx_quant((torch.randn((n, k), device="cuda") * 0.02).to(torch.bfloat16))
    b, b_scales = codes.t().contiguous(), scales.view(n, k // 64, 2).permute(1, 0, 2).contiguous()
    c = torch.empty((m, n), dtype=torch.bfloat16, device="cuda")
    symm = capi.symm_alloc(capi.symm_bytes_needed(capi.make_tiling(m, k, n, 1), False))
    for call in (lambda: capi.mx_quant_allgather_matmul(x, b, b_scales, c, symm, 1),
                 lambda: capi.mx_gemm(*capi.mx_quant(x), b, b_scales, out=c)):
        capi.trace_arm()
        call()
        table = timeline.summarise(capi.trace_read())
        assert table["ctas"] >= 1 and table["last tile committed"][0] > 0 and table["CTA end"][0] > 0, table
print("timeline ok")
"""


def test_one_rank_calls_leave_a_timeline():
    if not os.path.exists(os.path.join(ROOT, "catccos_b200", "libcatccos_b200_trace.so")):
        pytest.skip("needs the trace build: python -m catccos_b200.build --trace")
    out = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, env={**os.environ, "CATCCOS_B200_TRACE": "1"}, timeout=300,
                         capture_output=True, text=True)
    assert out.returncode == 0 and "timeline ok" in out.stdout, out.stdout + out.stderr

"""GPU test of what the calls on torch tensors take and raise."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def test_no_room_for_the_outputs_is_torch_out_of_memory(capi, cuda):
    # a program that serves near the limit catches torch.OutOfMemoryError and sheds load
    torch = cuda
    x = torch.zeros((8192, 32768), dtype=torch.bfloat16, device="cuda")  # 512 MiB; its codes take 256
    capi.mx_quant(x[:32])
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (64 << 20)) / total)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            capi.mx_quant(x)
        with pytest.raises(torch.OutOfMemoryError):
            capi.mx_gemm_quant_out(x.view(torch.uint8)[:, :128], x, x, x.view(64, 65536, 64))
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    codes, scales = capi.mx_quant(x[:32])
    assert codes.shape == (32, 32768) and scales.shape == (32, 1024)


def test_forms_of_a_symmetric_address(capi, cuda):
    torch = cuda
    x = torch.ones((16, 128), dtype=torch.bfloat16, device="cuda")
    codes, scales = capi.mx_quant(x)
    b, b_scales = torch.full((128, 16), 0x38, dtype=torch.uint8, device="cuda"), torch.full((2, 16, 2), 127, dtype=torch.uint8, device="cuda")
    symm = capi.symm_alloc(capi.symm_bytes_needed(capi.make_tiling(16, 128, 16, 1), False))
    try:
        for form in (symm, ctypes.c_void_p(symm)):
            c = torch.zeros((16, 16), dtype=torch.bfloat16, device="cuda")
            capi.mx_quant_allgather_matmul(x, b, b_scales, c, form, 1)
            assert bool((c == 128).all())  # 128 products of 1 and 1
            out = [torch.zeros_like(codes), torch.zeros_like(scales)]
            capi.mx_quant_allgather(x, *out, form, 1)
            assert torch.equal(out[0], codes) and torch.equal(out[1], scales)
        capi.mx_quant_allgather(x, *out, None, 1)  # one rank needs no symmetric buffer here
        capi.mx_quant_allgather(x, *out, ctypes.c_void_p(), 1)
        for bad in ("0", 1.5, c):
            with pytest.raises(TypeError):
                capi.mx_quant_allgather(x, *out, bad, 1)
    finally:
        capi.symm_free(symm)

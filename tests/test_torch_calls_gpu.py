"""GPU test of what the calls on torch tensors raise."""
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
